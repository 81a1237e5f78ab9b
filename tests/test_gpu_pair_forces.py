"""Pair forces and energy against the CPU oracle at ion counts around the edges of the kernel's
tiling: one ion pair, one and two ions past a block of 32, and both sides of the counts at which
the super-blocks grow from 2 to 4 (4225 ions) and from 4 to 8 blocks (8449), with a last block
of one ion. 1e-12 of the largest force: each is a sum of up to 8448 terms, a few rounding
errors each; 1e-10 of the energy, whose terms cancel."""
import numpy as np
import pytest

from maze_poisson_b200 import systems
from maze_poisson_b200.c_api import CAPI
from mdparity import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_ions,pot", [(2, 0), (33, 0), (66, 0), (4224, 0), (4225, 0), (8448, 0), (8449, 0),
                                        (33, 1), (4225, 1), (8449, 1), (33, 2), (4225, 2), (8449, 2)])
def test_tile_edges(product_path, oracle_path, n_ions, pot):
    s = systems.make_melt(n_ions + n_ions % 2, 32, seed=5)
    params = (s.pot_params, systems.lj_params_au(), systems.sc_params_au())[pot]
    out = []
    for lib in (CAPI(product_path), CAPI(oracle_path, extensions=False)):
        lib.solver_initialize()
        try:
            lib.solver_initialize_grid(32, s.L, s.h, 1e-7, 1.0, 1.0, 0, 0)
            lib.solver_initialize_particles(32, 2, s.L, s.h, n_ions, pot, 0, s.types[:n_ions].copy(),
                                            s.pos[:n_ions].copy(), s.vel[:n_ions].copy(), s.mass[:n_ions].copy(),
                                            s.charges[:n_ions].copy(), params)
            e, f = lib.solver_compute_forces_noel(), np.empty((n_ions, 3))
            lib.get_fcs_noel(f)
            out.append((e, f))
        finally:
            lib.solver_finalize()
    (e, f), (eo, fo) = out
    assert rel(f, fo) < 1e-12
    assert abs(e - eo) <= 1e-10 * abs(eo)
