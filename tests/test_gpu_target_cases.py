"""GPU test of the pixel mapping where its special cases lie: planes turned by
multiples of 90 degrees put whole rows and columns of pixels on phi = 0, 90 and
180 degrees and one on the pole; without a tilt the slant terms are zero.
Against the oracle's FP64 mapping.

Tolerance: the FP32 chain's allowance in the reprojection, eight units of the last
place of a unit cosine (2^-21 each) in pixels, 8 x 4.77e-7 / cell.
"""
import math

import numpy as np
import pytest

import fastimagingpipe_b200 as fip
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("turn", [0, 1, 2, 3])
@pytest.mark.parametrize("tilt", [0.0, 0.2])
@pytest.mark.parametrize("n,cell", [(16, 2e-3), (128, 7e-4)])
def test_targets_on_the_axes(cuda, n, cell, tilt, turn):
    import torch
    c, s = ((1, 0), (0, 1), (-1, 0), (0, -1))[turn]
    ct, st = math.cos(tilt), math.sin(tilt)
    V = np.array([c, s * ct, s * st, -s, c * ct, c * st, 0.0, -st, ct], np.float32)
    want = np.asarray(oracle.pixel_targets(V, n, cell, "f64")).reshape(n, n, 2)
    out = torch.zeros(n * n * 2, device=cuda)
    with fip.Imager(n, 16, cell, 0) as im:
        for evaluated in (False, True):
            im.pixel_targets(torch.tensor(V, device=cuda), out, evaluated=evaluated)
            got = out.cpu().numpy().reshape(n, n, 2)
            assert np.abs(got - want).max() <= 8 * 4.77e-7 / cell
