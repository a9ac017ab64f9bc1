"""GPU test of the precision form's reprojection by destination pixel (images
from 768 pixels a side) against the FP64 oracle: ragged sides, planes turned
and tilted by several hour angles and declinations, cells on both sides of the
plan's curvature limits (finer steps above 9e-6, the splat above 4.5e-5).

Tolerance: the precision form's bar for FP32 storage, 3e-5 relative RMS; the
reprojection's own share is below 1e-5 pixel of position, 1e-5 relative.
"""
import numpy as np
import pytest

import fastimagingpipe_b200 as fip
from fastimagingpipe_b200 import synthetic
import oracle

pytestmark = pytest.mark.gpu


def relrms(a, b):
    return float(np.sqrt(((a - b) ** 2).mean() / (b ** 2).mean()))


@pytest.mark.parametrize("n,cell,ha,dec", [
    (768, 1e-6, 1.5, -30.0), (772, 2e-5, 0.1, -27.0), (1000, 3e-5, 3.0, -30.0),
    (1028, 1.2e-5, -2.0, -60.0), (1028, 3.9e-5, 5.0, -10.0), (1024, 6e-5, 4.0, -30.0),
    (900, 2.5e-5, -4.5, 20.0)])
def test_pull_matches_fp64(cuda, n, cell, ha, dec):
    import torch
    snap = synthetic.make_snapshots(n_ant=40, radius_m=0.06 / cell, image_size=n, cell_size=cell,
                                    unit_size=20, hour_angle0_h=ha, dec_deg=dec, seed=n)
    nb = snap.num_baselines
    _, images, _ = oracle.fipipe(snap, "f64", want_images=True)
    d = {k: torch.tensor(getattr(snap, k), device=cuda) for k in ("vis_re", "vis_im", "B", "V")}
    img, mx = torch.zeros(n, n, device=cuda), torch.zeros(1, device=cuda)
    with fip.Imager(n, nb, cell, 20, form=fip.FORM_PRECISE) as im:
        for k in range(3):
            im.image_snapshot(d["vis_re"][k * nb:], d["vis_im"][k * nb:], d["B"][2 * k * nb:],
                              d["V"][9 * k:], nb, img, mx)
            got = img.cpu().numpy().astype(np.float64)
            want = np.asarray(images[k], np.float64).reshape(n, n)
            assert relrms(got, want) <= 3e-5
            assert abs(float(mx) - float(img.max())) == 0.0
        im.check()


@pytest.mark.parametrize("storage", [fip.STORE_F16, fip.STORE_BF16])
def test_image_of_nan_pixels_is_zero(cuda, storage):
    """An infinite visibility leaves NaN in every corrected pixel: the splat's
    integer sums image those as zero, and so does the pull."""
    import torch
    n, cell = 768, 3e-5
    snap = synthetic.make_snapshots(n_ant=24, radius_m=0.06 / cell, image_size=n, cell_size=cell,
                                    unit_size=32, n_snap=1, seed=3)
    d = {k: torch.tensor(getattr(snap, k), device=cuda) for k in ("vis_re", "vis_im", "B", "V")}
    d["vis_re"][5] = float("inf")
    img, mx = torch.ones(n, n, device=cuda), torch.ones(1, device=cuda)
    with fip.Imager(n, snap.num_baselines, cell, 32, form=fip.FORM_PRECISE,
                    vis_storage=storage) as im:
        im.image_snapshot(d["vis_re"], d["vis_im"], d["B"], d["V"], snap.num_baselines, img, mx)
    assert float(img.abs().max()) == 0.0 and float(mx) == 0.0
