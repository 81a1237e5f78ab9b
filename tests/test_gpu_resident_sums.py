"""Scalar products of the resident CG kernel (csrc/resident.cu) that shrink or grow by many
orders of magnitude from one iteration to the next: right-hand sides made of one or two
eigenvectors of the operator, whose residual collapses to rounding within one or two iterations.

Bounds: an eigenvector's solution is known, x = b / lambda; the solver leaves a residual of at
most tol, which the smallest eigenvalue turns into an error of x, and FP64 adds about
1e-15 * 12 max|x| to the residual (12: the largest eigenvalue). Both are held with a factor of
ten. Iteration counts are not compared: after the collapse they are the rounding's."""
import numpy as np
import pytest

from maze_poisson_b200.c_api import CAPI

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(product_path):
    c = CAPI(product_path)
    c.solver_initialize()
    return c


def plane_wave(n):
    """cos(2 pi i / n) and its eigenvalue under the periodic 7-point Laplacian."""
    wave = np.cos(2 * np.pi * np.arange(n) / n)[:, None, None] * np.ones((n, n, n))
    return wave, 2 * np.cos(2 * np.pi / n) - 2


def check(it, x, exact, residual, tol, smallest):
    assert np.isfinite(x).all() and it >= 0
    top = np.max(np.abs(exact))
    assert residual <= tol + 1e-14 * 12 * top
    # the solver is free to add a constant where the operator is singular
    assert np.max(np.abs((x - x.mean()) - exact)) <= 10 * (tol / abs(smallest) + 1e-14 * top * 12 / abs(smallest))


@pytest.mark.parametrize("precond", [0, 1])
@pytest.mark.parametrize("n,amplitude,tol", [(16, 1e6, 1e-10), (32, 1e2, 1e-12), (32, 1e4, 1e-10), (32, 1e6, 1e-10),
                                             (64, 1e6, 1e-8)])
def test_sum_collapses(lib, oracle_lib, n, amplitude, tol, precond):
    wave, lam = plane_wave(n)
    b = np.ascontiguousarray(amplitude * wave)
    x, lx = np.empty_like(b), np.empty_like(b)
    it = lib.mzb_conj_grad(b, np.zeros_like(b), x, tol, n, precond)
    oracle_lib.orc_laplace(x, lx, n)
    check(it, x, b / lam, np.max(np.abs(lx - b)), tol, lam)


@pytest.mark.parametrize("n,amplitude,tol", [(32, 1e6, 1e-9), (66, 1e4, 1e-10)])
def test_sum_collapses_pb(lib, oracle_lib, n, amplitude, tol):
    """Uniform coefficients: the eigenvector's value is 3 lambda - 0.25."""
    wave, lam = plane_wave(n)
    lam = 3.0 * lam - 0.25
    b = np.ascontiguousarray(amplitude * wave)
    e, k2 = [np.full((n, n, n), 3.0) for _ in range(3)], np.full((n, n, n), 0.25)
    x, lx = np.empty_like(b), np.empty_like(b)
    it = lib.mzb_conj_grad_pb(b, np.zeros_like(b), x, tol, n, *e, k2)
    oracle_lib.orc_laplace_pb(x, lx, *e, k2, n)
    check(it, x, b / lam, np.max(np.abs(lx - b)), tol, -0.25)


def test_sum_grows_then_collapses(lib, oracle_lib):
    """The lowest and the highest mode, weighted so that <p, A p> grows by more than 2^20 in the
    second iteration (past the fixed-point words' range) and the residual then vanishes."""
    n, tol = 96, 1e-11
    wave, low = plane_wave(n)
    i = np.arange(n)
    checker = 1.0 - 2.0 * ((i[:, None, None] + i[None, :, None] + i[None, None, :]) % 2)
    share = np.sqrt(0.5 * abs(low) / 12)
    b = np.ascontiguousarray(1e2 * (wave + share * checker))
    exact = 1e2 * (wave / low + share * checker / -12.0)
    x, lx = np.empty_like(b), np.empty_like(b)
    it = lib.mzb_conj_grad(b, np.zeros_like(b), x, tol, n, 0)
    oracle_lib.orc_laplace(x, lx, n)
    check(it, x, exact, np.max(np.abs(lx - b)), tol, low)
