"""GPU test of the long run-time-length transforms against FP64 steps from the same
grid: a codelet-only length, prime factors of 251 to 509, the longest length and the
first sides beyond it (cuFFT).

Tolerance: 2.3e-6 relative RMS as for the steps from the grid to the image of other
sides (targets of the reprojection 2.0e-6, transform and correction 1e-6), and a
prime pass's sums of up to 254 products, 2^-24 x sqrt(254) = 1e-6, in quadrature:
2.5e-6, 3e-6 with a margin.  The outermost pixels are left out: a source whose
target lies within FP32's rounding of the edge (1e-4 pixel at these sides) may be
dropped or kept, as in the reference.
"""
import pytest

from test_gpu_pull_accuracy import after_grid_error

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3000, 3012, 3032, 4072, 4796, 4800, 4804, 4832, 5000])
def test_long_lengths_match_fp64(cuda, n):
    assert after_grid_error(cuda, n, 7.2722e-6 * 4096 / n, 1.5, -30.0, border=2) <= 3e-6
