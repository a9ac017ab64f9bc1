"""GPU test of the reduced storage in calls that share launches over their snapshots:
counts that differ by samples or by whole blocks of 1,024 take as many launches as
equal ones, and the tLISI agrees with snapshots imaged one by one (1e-5 absolute:
the same kernels)."""
import numpy as np
import pytest

import fastimagingpipe_b200 as fip
from fastimagingpipe_b200 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", [fip.STORE_F16, fip.STORE_BF16])
@pytest.mark.parametrize("cut", [(0, 0, 0, 0), (1, 0, 13, 7), (0, 1024, 4000, 4949)])
def test_uneven_counts_share_a_conversion(cuda, storage, cut):
    import torch
    n, t, cell = 256, 16, 4e-5
    s = synthetic.make_snapshots(n_ant=100, radius_m=800.0, image_size=n, cell_size=cell,
                                 unit_size=t, n_snap=4, seed=5)
    nb = s.num_baselines
    counts = [nb - c for c in cut]
    d = {k: torch.tensor(getattr(s, k), device=cuda) for k in ("vis_re", "vis_im", "B", "V")}
    kw = dict(form=fip.FORM_PRECISE, vis_storage=storage)
    got = torch.zeros(2, (n // t) ** 2, device=cuda)
    even = torch.zeros_like(got)
    with fip.Imager(n, nb, cell, t, **kw) as im:
        im.image_sequence(d["vis_re"], d["vis_im"], d["B"], d["V"], [nb] * 4, nb, even)
        per_call = im.kernel_launches
        im.image_sequence(d["vis_re"], d["vis_im"], d["B"], d["V"], counts, nb, got)
        assert im.kernel_launches == 2 * per_call
    imgs, mx = torch.zeros(4, n, n, device=cuda), torch.zeros(4, device=cuda)
    want = torch.zeros_like(got)
    with fip.Imager(n, nb, cell, t, **kw) as im:
        for k in range(4):
            im.image_snapshot(d["vis_re"][k * nb:], d["vis_im"][k * nb:], d["B"][2 * k * nb:],
                              d["V"][9 * k:], counts[k], imgs[k], mx[k:])
        for k in range(2):
            im.trigger(imgs[k], imgs[k + 1], imgs[k + 2], mx[k:], want[k])
        torch.cuda.synchronize()
    assert np.abs(got.cpu().numpy() - want.cpu().numpy()).max() <= 1e-5
