"""CG iterates after a given number of iterations, odd and even, against the CPU oracle: the
resident kernel (x in tensor memory and in the grid) and the streaming one, whose x lags a
direction behind in every second iteration.

The oracle stops at some tolerance; the tolerance handed to the library is that residual's
own maximum and a little more, so both stop at the same iteration and x is compared there.
The iterates differ only through the order of the scalar products' sums (about 1e-15 each, a
handful of iterations): 1e-12 of the largest value."""
import numpy as np
import pytest

from maze_poisson_b200.c_api import CAPI

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(product_path):
    c = CAPI(product_path)
    c.solver_initialize()
    return c


@pytest.mark.parametrize("n,precond", [(16, 0), (64, 1), (106, 0), (128, 1), (144, 1), (208, 0), (240, 0), (256, 1)])
def test_iterates(lib, oracle_lib, n, precond):
    rng = np.random.default_rng(n)
    b = rng.standard_normal((n, n, n))
    b -= b.mean()
    x0 = 0.1 * rng.standard_normal((n, n, n))
    x, xo, lx = np.empty_like(b), np.empty_like(b), np.empty_like(b)
    tol, seen = 1.0, set()
    while len(seen) < 2:
        tol *= 0.7
        assert tol > 1e-3
        its = oracle_lib.orc_conj_grad(b, x0, xo, tol, n)
        if its < 3 or its % 2 in seen:
            continue
        oracle_lib.orc_laplace(xo, lx, n)
        stop = np.max(np.abs(lx - b)) * (1 + 1e-6)
        assert lib.mzb_conj_grad(b, x0, x, stop, n, precond) == its
        assert np.max(np.abs(x - xo)) < 1e-12 * np.max(np.abs(xo)), its
        seen.add(its % 2)
