"""GPU test of calls whose snapshots share launches (images up to 1024 pixels a
side) against one snapshot at a time: three-snapshot calls, and sequences of
every remainder modulo the three-snapshot groups with uneven counts.

Both sides sum the same taps; only the order of FP32 additions into split grid
tiles differs (a few 2^-24 of a cell), so images agree to 1e-6 relative RMS
and tLISI (1 minus a product of tile means) to 1e-6.
"""
import numpy as np
import pytest

import fastimagingpipe_b200 as fip
from fastimagingpipe_b200 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [{}, dict(form=fip.FORM_PRECISE),
                                dict(form=fip.FORM_PRECISE, vis_storage=fip.STORE_F16)])
@pytest.mark.parametrize("n,ns,uneven", [(64, 3, False), (64, 4, True), (128, 5, True),
                                         (1024, 7, True), (1024, 6, False), (2048, 4, True)])
def test_shared_launches_match_single_snapshots(cuda, n, ns, uneven, kw):
    import torch
    t = 16
    snap = synthetic.make_snapshots(n_ant=64, radius_m=400.0, image_size=n, cell_size=0.015 / n,
                                    unit_size=t, n_snap=ns, transient_snapshot=ns - 1, seed=n + ns)
    nb, u = snap.num_baselines, n // t
    nbs = [nb - (97 * k if uneven else 0) for k in range(ns)]
    d = {k: torch.tensor(getattr(snap, k), device=cuda) for k in ("vis_re", "vis_im", "B", "V")}
    with fip.Imager(n, nb, snap.cell_size, t, **kw) as im:
        imgs = torch.zeros(ns, n, n, device=cuda)
        mx = torch.zeros(ns, device=cuda)
        for k in range(ns):
            im.image_snapshot(d["vis_re"][k * nb:], d["vis_im"][k * nb:], d["B"][2 * k * nb:],
                              d["V"][9 * k:], nbs[k], imgs[k], mx[k:])
        want = torch.zeros(ns - 2, u * u, device=cuda)
        for k in range(ns - 2):
            im.trigger(imgs[k], imgs[k + 1], imgs[k + 2], mx[k:], want[k])
        got = torch.zeros(ns - 2, u * u, device=cuda)
        im.image_sequence(d["vis_re"], d["vis_im"], d["B"], d["V"], nbs, nb, got)
        assert float((got - want).abs().max()) <= 1e-6
        if not uneven:
            one = torch.zeros(u * u, device=cuda)
            for _ in range(2):  # the second call on used scratch
                im.pipe_device(d["vis_re"], d["vis_im"], d["B"], d["V"], nb, one)
            assert float((one - want[0]).abs().max()) <= 1e-6
            host = im.pipe_host(*(a.cpu().numpy() for a in d.values()), nb, ns)
            assert np.abs(host.reshape(-1) - want[0].cpu().numpy()).max() <= 1e-6
