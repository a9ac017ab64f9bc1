"""GPU test of the run-time-length transform (image sides that are multiples of
four but not powers of two) against the FP64 oracle: every codelet radix, prime
factors with passes of their own, one- to five-pass lengths, bands wider than
a third of the grid and up to its edge, and one prime factor beyond the limit
(cuFFT).

Precision form, FP32 storage.  Tolerance 3e-5 relative RMS, the form's bar;
the transform's share is a few 2^-24 per pass.
"""
import numpy as np
import pytest

import fastimagingpipe_b200 as fip
from fastimagingpipe_b200 import synthetic
import oracle

pytestmark = pytest.mark.gpu


def relrms(a, b):
    return float(np.sqrt(((a - b) ** 2).mean() / (b ** 2).mean()))


@pytest.mark.parametrize("n", [20, 24, 28, 36, 48, 60, 72, 80, 84, 96, 100, 120, 140, 144, 180,
                               196, 240, 300, 324, 360, 384, 500, 44, 52, 68, 76, 484, 572, 604,
                               788, 796, 844, 1004])
@pytest.mark.parametrize("reach", [0.2, 0.62, 1.0])
def test_lengths_match_fp64(cuda, n, reach):
    import torch
    cell = 0.012 / n
    # Longest baseline (wavelengths) as a share of the grid's half side, 1 / (2 cell).
    radius = reach * 0.5 / cell * (299792458.0 / 140e6) / 2
    snap = synthetic.make_snapshots(n_ant=30, radius_m=radius, image_size=n, cell_size=cell,
                                    unit_size=4, seed=n)
    nb = snap.num_baselines
    _, images, _ = oracle.fipipe(snap, "f64", want_images=True)
    d = {k: torch.tensor(getattr(snap, k), device=cuda) for k in ("vis_re", "vis_im", "B", "V")}
    img = torch.zeros(n, n, device=cuda)
    with fip.Imager(n, nb, cell, 4, form=fip.FORM_PRECISE) as im:
        for k in (0, 2):
            im.image_snapshot(d["vis_re"][k * nb:], d["vis_im"][k * nb:], d["B"][2 * k * nb:],
                              d["V"][9 * k:], nb, img)
            assert relrms(img.cpu().numpy().astype(np.float64), images[k]) <= 3e-5
        im.set_tuning(16)  # no shapes to choose from at these lengths
        assert im.tuning()["fft_values_per_thread"] == 0
