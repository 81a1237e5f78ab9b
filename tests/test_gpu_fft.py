"""The FFT Poisson solve at every factor split of the register-resident passes (csrc/fft.cu:
N1 a multiple of N2 and not, rows inside a warp and across warps) and at the sizes beside
them that the shared-memory kernels keep, against numpy. 1e-12 of the field's maximum, the
bound of the other FFT tests: both sides are FP64 transforms of at most 288 points per line
with rounding errors of a few 1e-16."""
import numpy as np
import pytest

from maze_poisson_b200.c_api import CAPI
from oracle.fft_oracle import fft_poisson

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [24, 27, 32, 36, 48, 54, 64, 72, 81, 96, 108, 128, 144, 162, 192, 216, 256, 288])
def test_fft_sizes(product_path, n):
    c = CAPI(product_path)
    c.solver_initialize()
    q = np.random.default_rng(n).standard_normal((n, n, n))
    phi, L = np.empty_like(q), 0.3 * n
    c.mzb_fft_poisson(q, phi, n, L, L / n)
    ref = fft_poisson(q, L, L / n)
    assert np.max(np.abs(phi - ref)) < 1e-12 * np.max(np.abs(ref))
