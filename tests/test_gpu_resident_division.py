"""The Jacobi preconditioner's r / 6 in the resident CG kernel, a product and one exact remainder
instead of a division, rounds as the division does: a right-hand side with one value in one
point makes every scalar product a single term, so x after the first iteration must be NumPy's
to the last bit."""
import numpy as np
import pytest

from maze_poisson_b200.c_api import CAPI

pytestmark = pytest.mark.gpu


def first_iterate(r):
    p = r / 6.0
    alpha = (r * -p) / (p * -(p * 6.0))
    return alpha * p


def values():
    rng = np.random.default_rng(6)
    near = np.array([3.0, 6.0, 9.0, 1.0 + 2.0 ** -52, 6.0 - 2.0 ** -50, 7.0, 11.0, 2.0 ** 53 - 1, 2.0 ** -60])
    wide = rng.standard_normal(300) * 10.0 ** rng.uniform(-90, 90, 300)
    return np.concatenate([near, -near, rng.integers(1, 2 ** 53, 100).astype(float), wide])


def test_sixth(product_path):
    lib = CAPI(product_path)
    lib.solver_initialize()
    n = 16
    b, x0, x = (np.zeros((n, n, n)) for _ in range(3))
    for r in values():
        b[3, 4, 5] = -r
        assert lib.mzb_conj_grad(b, x0, x, abs(r), n, 1) == 0
        assert x[3, 4, 5] == first_iterate(r), r
        assert np.count_nonzero(x) == 1
