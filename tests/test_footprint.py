"""mzb_system_footprint, the bytes by which jobs are admitted against the memory budget."""
import ctypes

import pytest

MB = 1024.0 * 1024.0


@pytest.fixture(scope="module")
def footprint(product_path):
    f = ctypes.CDLL(product_path).mzb_system_footprint
    f.restype = ctypes.c_double
    f.argtypes = [ctypes.c_int, ctypes.c_int]
    return f


def pair_partials(n_ions):
    """Bytes of the pair forces' partial sums: two sides of every pair of super-blocks, sb blocks
    of 32 ions each, sb the largest of 8, 4 and 2 that gives 592 pairs."""
    blocks = -(-n_ions // 32)
    for sb in (8, 4, 2):
        super_blocks = -(-blocks // sb)
        pairs = super_blocks * (super_blocks + 1) // 2
        if pairs >= 592:
            break
    return pairs * 2 * sb * 32 * 3 * 8


# the work area of the resident solves on 148 SMs: a CTA's eight halo strips, 16 bytes a value
HALO = {64: 11 * 13 * 8 * 6 * 64 * 16, 116: 5 * 29 * 8 * 24 * 116 * 16, 128: 9 * 16 * 8 * 15 * 128 * 16, 192: 0}


@pytest.mark.parametrize("n", sorted(HALO))
def test_grid_side(footprint, n):
    """Ten grids, the resident solves' work area and the constant part; at most the multigrid
    levels' 3 * 4 * 8 / 7 bytes a point and a few MB beside them."""
    least = 10 * 8 * n ** 3 + HALO[n] + 64 * MB
    assert least <= footprint(n, 0) <= least + 14 * n ** 3 + 4 * MB


@pytest.mark.parametrize("n_ions", [1000, 4224, 4225, 8448, 8449, 16000])
def test_ion_side(footprint, n_ions):
    """Seven vectors, the spline weights and the pair forces' partial sums."""
    least = n_ions * (7 * 24 + 12 * 8) + pair_partials(n_ions) - pair_partials(1)
    assert least <= footprint(64, n_ions) - footprint(64, 0) <= 1.1 * least + 100 * n_ions


@pytest.mark.gpu
@pytest.mark.parametrize("n,n_ions,cas", [(116, 250, "cic"), (64, 8448, "spl_cubic")])
def test_holds_what_a_system_takes(product_path, n, n_ions, cas):
    import torch

    from maze_poisson_b200 import systems
    from maze_poisson_b200.c_api import CAPI
    from maze_poisson_b200.md import MDRun

    lib = CAPI(product_path)
    lib.solver_initialize()
    warm = lib.mzb_system_create()
    run = MDRun(lib, systems.make_melt(64, 16, seed=1), method="LCG", precision=1)
    run.initialize()
    run.step()
    lib.mzb_system_destroy(warm)
    lib.mzb_trim_device_cache()
    free = torch.cuda.mem_get_info()[0]
    handle = lib.mzb_system_create()
    run = MDRun(lib, systems.make_melt(n_ions, n, seed=1), method="LCG", precision=1, cas=cas)
    run.initialize()
    run.step()
    used = free - torch.cuda.mem_get_info()[0]
    lib.mzb_system_destroy(handle)
    lib.mzb_trim_device_cache()
    assert 0 < used <= lib.mzb_system_footprint(n, n_ions)
