"""The pair-force kernel's 1/r to a few units in the last place: two ions under the soft-core
potential with nu = d = B = 1, whose force is 1/r^2 - 1/r_cut^2, at separations over the
whole range, against 80-bit arithmetic. Coordinates are dyadic, so the separation itself is exact.

Bound, in units of 2^-53: r^2 3, so r 1.5; 1/r 2 more (two fused steps, the last one's rounding
included); d / r 1, pow 4 (2 ulp), so 8.5; (1/r)^2 8; their product, the shift and the
component 2: below 20 of the two terms' sum. 24 is allowed."""
import numpy as np
import pytest

from maze_poisson_b200 import systems
from maze_poisson_b200.c_api import CAPI

pytestmark = pytest.mark.gpu
L = 64.0


def separations():
    rng = np.random.default_rng(7)
    out = []
    for r in np.geomspace(2e-3, 0.49 * L, 160):
        v = rng.standard_normal(3)
        v *= r / np.linalg.norm(v)
        out.append(np.round(v * 2.0 ** 40) / 2.0 ** 40)
    return out


def test_inverse_distance(product_path):
    lib = CAPI(product_path)
    s = systems.make_melt(64, 32, seed=1)
    rc = np.longdouble(L / 2)
    u = np.longdouble(2.0) ** -53
    worst = 0.0
    lib.solver_initialize()
    try:
        lib.solver_initialize_grid(32, L, L / 32, 1e-7, 1.0, 1.0, 0, 0)
        for v in separations():
            pos = np.full((2, 3), 32.0)
            pos[1] += v
            lib.solver_initialize_particles(32, 2, L, L / 32, 2, 2, 0, s.types[:2].copy(), pos, np.zeros((2, 3)),
                                            s.mass[:2].copy(), s.charges[:2].copy(), np.ones(3))
            lib.solver_compute_forces_noel()
            f = np.empty((2, 3))
            lib.get_fcs_noel(f)
            d = (pos[0] - pos[1]).astype(np.longdouble)
            r2 = np.sum(d * d)
            r = np.sqrt(r2)
            main, shift = d / (r2 * r), d / (rc * rc * r)
            err = np.abs(f[0].astype(np.longdouble) - (main - shift)) / (np.abs(main) + np.abs(shift))
            assert np.array_equal(f[1], -f[0])
            worst = max(worst, float(np.max(err) / u))
    finally:
        lib.solver_finalize()
    print(f"largest error of a force component: {worst:.1f} 2^-53")
    assert worst < 24
