"""The resident CG kernel (csrc/resident.cu) against the CPU oracle at the sizes where its
layout changes: the smallest grid, uneven patches, one and two pairs of a row per lane
(n = 64, 66), x in tensor memory and in the grid (10 and more pairs per thread, n = 104 and
116), the largest grid.

Tolerances: the iterates differ from the oracle's only through the order of the scalar
products' sums (about 1e-15 each), so the iteration counts agree within 1 and, where they are
equal, the solutions within 1e-10, the bound of the other FP64 solves; a solution's residual
meets the solver's tolerance up to the rounding between the recursive and the true residual.
"""
import numpy as np
import pytest

import mdparity
from maze_poisson_b200.c_api import CAPI
from maze_poisson_b200.systems import make_melt, make_pb_system, pb_settings

pytestmark = pytest.mark.gpu
TOL = 1e-6


@pytest.fixture(scope="module")
def lib(product_path):
    c = CAPI(product_path)
    c.solver_initialize()
    return c


def rel(a, b):
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


def problem(n, oracle_lib, coefficients=None):
    rng = np.random.default_rng(n)
    xt, x0 = rng.standard_normal((n, n, n)), 0.1 * rng.standard_normal((n, n, n))
    b = np.empty_like(xt)
    if coefficients is None:
        oracle_lib.orc_laplace(xt, b, n)
    else:
        oracle_lib.orc_laplace_pb(xt, b, *coefficients, n)
    return b, x0


@pytest.mark.parametrize("n,precond", [(16, 0), (18, 1), (34, 0), (50, 1), (64, 0), (66, 1), (90, 0), (104, 1),
                                       (106, 0), (116, 1), (128, 0)])
def test_cg_sizes(lib, oracle_lib, n, precond):
    b, x0 = problem(n, oracle_lib)
    x, xo, lx = np.empty_like(b), np.empty_like(b), np.empty_like(b)
    it = lib.mzb_conj_grad(b, x0, x, TOL, n, precond)
    ito = oracle_lib.orc_conj_grad(b, x0, xo, TOL, n)
    assert abs(it - ito) <= 1
    if it == ito:
        assert rel(x, xo) < 1e-10
    oracle_lib.orc_laplace(x, lx, n)
    assert np.max(np.abs(lx - b)) <= TOL * (1 + 1e-6)


@pytest.mark.parametrize("n", [16, 50, 66, 106, 128])
def test_cg_pb_sizes(lib, oracle_lib, n):
    """Coefficients equal to the grid corner's in most rows (those pairs take the constants),
    random ones elsewhere."""
    rng = np.random.default_rng(100 + n)
    e = [np.full((n, n, n), 3.0) for _ in range(3)]
    k2 = np.full((n, n, n), 0.25)
    box = slice(n // 3, n // 2 + 1)
    for a in e:
        a[box, box, box] = 1.0 + 2.0 * rng.random((n, n, n))[box, box, box]
    k2[box, box, box] = 0.0
    b, x0 = problem(n, oracle_lib, (*e, k2))
    x, xo, lx = np.empty_like(b), np.empty_like(b), np.empty_like(b)
    it = lib.mzb_conj_grad_pb(b, x0, x, TOL, n, *e, k2)
    ito = oracle_lib.orc_conj_grad_pb(b, x0, xo, TOL, n, *e, k2)
    assert abs(it - ito) <= 1
    if it == ito:
        assert rel(x, xo) < 1e-10
    oracle_lib.orc_laplace_pb(x, lx, *e, k2, n)
    assert np.max(np.abs(lx - b)) <= TOL * (1 + 1e-6)


@pytest.mark.parametrize("power", [-490, 490])
def test_cg_out_of_fixed_point_range(lib, oracle_lib, power):
    """Scaled by 2^+-490 the scalar products leave the range of the fixed-point sums and go
    through the partials; everything else scales exactly."""
    n, s = 32, 2.0 ** power
    b, x0 = problem(n, oracle_lib)
    x, y = np.empty_like(b), np.empty_like(b)
    it = lib.mzb_conj_grad(b, x0, x, TOL, n, 0)
    assert abs(lib.mzb_conj_grad(b * s, x0 * s, y, TOL * s, n, 0) - it) <= 1
    assert rel(y / s, x) < 1e-5
    assert np.isfinite(y).all()


@pytest.mark.parametrize("n,ions,method,pb", [(32, 128, "MULTIGRID", False), (64, 250, "MAZE-MULTIGRID", False),
                                              (68, 250, "MULTIGRID", False), (84, 432, "MAZE-MULTIGRID", False),
                                              (32, 8, "MAZE-MULTIGRID", True), (68, 8, "MULTIGRID", True)])
def test_multigrid_sizes(lib, oracle_path, n, ions, method, pb):
    """The resident multigrid kernel in MD steps: patches of the coarse grid that fill the
    CTAs and that leave some without, one and two pairs of a row per lane. The V-cycle amplifies
    the order of the coarse CG's sums, so the bound is five times the oracle's own change under
    a 1e-15 scaling of the positions, at least 1e-10."""
    orc = CAPI(oracle_path, extensions=False)
    kw = dict(method=method, tol=1e-10, integrator="VERLET")
    if pb:
        system = make_pb_system(ions, n, 0.5 * n, seed=n)
        kw.update(pb=pb_settings(system), eps_s=78.4, eps_int=1.0, T=300.0)
    else:
        system = make_melt(ions, n, seed=n)
    floor = mdparity.oracle_floor(orc, system, 2, **kw)
    bounds = {k: max(1e-10, 5 * floor["fcs_elec"], 5 * floor["fcs_tot"]) for k in ("fcs_elec", "fcs_tot", "vel")}
    mdparity.run_pair(lib, orc, system, 2, bounds=bounds, **kw)
