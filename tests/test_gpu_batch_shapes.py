"""GPU test of batches whose calls alternate between more shapes (snapshots per
sequence) than executable graphs are kept: every call's tLISI as from a batch
that takes one snapshot at a time (1e-6: only the order of FP32 additions into
split grid tiles differs)."""
import numpy as np
import pytest

import fastimagingpipe_b200 as fip
from fastimagingpipe_b200 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [{}, dict(form=fip.FORM_PRECISE, vis_storage=fip.STORE_F16)])
def test_alternating_call_shapes(cuda, kw):
    import torch
    calls = [1, 3, 2, 1, 3, 5, 4, 1, 6, 7, 8, 9, 10, 1, 3, 2]
    total = sum(calls)
    snap = synthetic.config_tiny(n_snap=6, transient_snapshot=4)
    nb, n, t = snap.num_baselines, snap.image_size, snap.unit_size
    u2 = (n // t) ** 2
    d = {k: torch.tensor(getattr(snap, k), device=cuda) for k in ("vis_re", "vis_im", "B", "V")}

    def args(ks):
        ks = [k % 6 for k in ks]
        return ([d["vis_re"][k * nb:] for k in ks], [d["vis_im"][k * nb:] for k in ks],
                [d["B"][2 * k * nb:] for k in ks], [d["V"][9 * k:] for k in ks], [nb] * len(ks))

    def results(sizes):
        out = torch.zeros(total, u2, device=cuda)
        done = at = 0
        with fip.Batch(n, nb, snap.cell_size, t, 10, **kw) as b:
            for c in sizes:
                done += b.image(*args(range(at, at + c)), out[done:])
                at += c
            torch.cuda.synchronize()
        assert done == total - 2
        return out[:done].cpu().numpy()

    assert np.abs(results(calls) - results([1] * total)).max() <= 1e-6
