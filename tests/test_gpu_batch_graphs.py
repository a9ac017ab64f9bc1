"""GPU test of a batch's kept graphs: calls of one shape (snapshots per sequence,
whether each triggers) share one executable graph, whatever their numbers of
triggers, and its updates take the new extents (tLISI as of one long call, 1e-5
absolute: the same kernels)."""
import numpy as np
import pytest

import fastimagingpipe_b200 as fip
from fastimagingpipe_b200 import synthetic

pytestmark = pytest.mark.gpu


def instantiations(call):
    """Graph instantiations that the CUDA runtime records during call()."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    return sum("cudaGraphInstantiate" in e.name for e in p.events())


@pytest.mark.parametrize("kw", [{}, dict(form=fip.FORM_PRECISE, vis_storage=fip.STORE_BF16)])
@pytest.mark.parametrize("count", [3, 4])  # one triple (no streaming) and two in the first call
def test_calls_of_one_shape_share_a_graph(cuda, count, kw):
    import torch
    sizes = (512, 256)
    cell = 2.9e-5
    data = []
    for n in sizes:
        s = synthetic.make_snapshots(n_ant=24, radius_m=800.0, image_size=n, cell_size=cell,
                                     unit_size=16, n_snap=2 * count, seed=n)
        nb = s.num_baselines
        d = {k: torch.tensor(getattr(s, k), device=cuda) for k in ("vis_re", "vis_im", "B", "V")}
        data.append([(d["vis_re"][k * nb:], d["vis_im"][k * nb:], d["B"][2 * k * nb:],
                      d["V"][9 * k:]) for k in range(2 * count)])
    seqs = [(n, nb, cell, 16) for n in sizes]

    def call(b, k0, k1, out):
        order = [(c, data[c][k]) for k in range(k0, k1) for c in range(2)]
        return b.image_sequences([c for c, _ in order], *([x[i] for _, x in order]
                                                          for i in range(4)),
                                 [nb] * len(order), out)

    out = lambda: [torch.zeros(2 * count, (n // 16) ** 2, device=cuda) for n in sizes]
    want, first, second, again = out(), out(), out(), out()
    with fip.Batch.of_sequences(seqs, 2 * count, **kw) as b:
        call(b, 0, 2 * count, want)
    with fip.Batch.of_sequences(seqs, count, **kw) as b:
        assert instantiations(lambda: call(b, 0, count, first)) == 1
        assert instantiations(lambda: call(b, count, 2 * count, second)) == 0
        b.reset()
        assert instantiations(lambda: call(b, 0, count, again)) == 0
    for c in range(2):
        w = want[c].cpu().numpy()
        for got, lo, hi in ((first, 0, count - 2), (second, count - 2, 2 * count - 2),
                            (again, 0, count - 2)):
            assert np.abs(got[c][:hi - lo].cpu().numpy() - w[lo:hi]).max() <= 1e-5
