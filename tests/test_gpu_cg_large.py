"""The streaming CG kernel (csrc/cg_fast.cu) above the resident kernel's sizes, at grids whose
cut differs: the fewest planes per block (n = 144), blocks of odd and even row counts (176,
208), uneven rows (240), all 148 SMs (256); several tolerances, so that solves end with and
without a direction that x still lacks. Against the CPU oracle up to 208, where iterates differ
only through the order of the scalar products' sums (1e-10, the bound of the other FP64
solves); the true residual meets the tolerance up to rounding."""
import numpy as np
import pytest

from maze_poisson_b200.c_api import CAPI

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(product_path):
    c = CAPI(product_path)
    c.solver_initialize()
    return c


@pytest.mark.parametrize("n,precond,tols", [(144, 0, (3.0, 1.0, 1e-2)), (176, 1, (1.0, 1e-1)), (208, 0, (1.0,)),
                                            (240, 1, (1.0, 1e-1)), (256, 0, (1.0, 5e-1, 1e-1))])
def test_cg_large(lib, oracle_lib, n, precond, tols):
    rng = np.random.default_rng(n)
    xt, x0 = rng.standard_normal((n, n, n)), 0.1 * rng.standard_normal((n, n, n))
    b, x, lx = np.empty_like(xt), np.empty_like(xt), np.empty_like(xt)
    oracle_lib.orc_laplace(xt, b, n)
    for tol in tols:
        it = lib.mzb_conj_grad(b, x0, x, tol, n, precond)
        oracle_lib.orc_laplace(x, lx, n)
        assert it > 0 and np.max(np.abs(lx - b)) <= tol * (1 + 1e-6)
        if n > 208:
            continue
        xo = np.empty_like(xt)
        ito = oracle_lib.orc_conj_grad(b, x0, xo, tol, n)
        assert abs(it - ito) <= 1
        if it == ito:
            assert np.max(np.abs(x - xo)) < 1e-10 * np.max(np.abs(xo))
