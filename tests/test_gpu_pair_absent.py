"""Pair forces with ions that are nowhere (a coordinate NaN, infinite or beyond 1e300): they take
part in no pair, and the other ions' forces and the energy are those of the system without
them. Bounds: the order of the sums changes with the ions' blocks, as in the tile-edge test
(1e-12 of the largest force, 1e-10 of the energy). Cells, blocks and pairs are indexed by clamped
integers, so such a coordinate addresses nothing."""
import numpy as np
import pytest

from maze_poisson_b200 import systems
from maze_poisson_b200.c_api import CAPI
from mdparity import rel

pytestmark = pytest.mark.gpu


def pair_forces(lib, s, pos, keep, pot, params):
    types, mass, charges = (a[keep].copy() for a in (s.types, s.mass, s.charges))
    x = np.ascontiguousarray(pos[keep])
    lib.solver_initialize_particles(32, 2, s.L, s.h, len(x), pot, 0, types, x, np.zeros_like(x), mass, charges, params)
    e, f = lib.solver_compute_forces_noel(), np.empty_like(x)
    lib.get_fcs_noel(f)
    return e, f


@pytest.mark.parametrize("pot", [0, 1, 2])
@pytest.mark.parametrize("n_ions", [34, 250, 4400])
def test_absent_ions(product_path, n_ions, pot):
    lib = CAPI(product_path)
    s = systems.make_melt(n_ions, 32, seed=3)
    params = (s.pot_params, systems.lj_params_au(), systems.sc_params_au())[pot]
    pos = s.pos.copy()
    lost = np.array([1, 2, n_ions // 2, n_ions - 3])
    for p, d, v in zip(lost, (0, 1, 2, 0), (np.nan, np.inf, -np.inf, 1e305)):
        pos[p, d] = v
    there = np.setdiff1d(np.arange(n_ions), lost)
    lib.solver_initialize()
    try:
        lib.solver_initialize_grid(32, s.L, s.h, 1e-7, 1.0, 1.0, 0, 0)
        eo, fo = pair_forces(lib, s, pos, there, pot, params)
        e, f = pair_forces(lib, s, pos, np.arange(n_ions), pot, params)
    finally:
        lib.solver_finalize()
    assert np.array_equal(f[lost], np.zeros((len(lost), 3)))
    assert rel(f[there], fo) < 1e-12
    assert abs(e - eo) <= 1e-10 * abs(eo)
