"""GPU test of the transient search over dense matrices: every location from one
launch whatever their number (no neighbouring two are minima, so ceil(u / 2)^2
records hold them all), in the order and with the values of the rule restated
in oracle.locate (positions to 1e-3 pixel: FP32 centroids)."""
import numpy as np
import pytest

import fastimagingpipe_b200 as fip
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("u,kind", [(129, "grid"), (256, "noise"), (511, "noise"),
                                    (512, "grid")])
def test_dense_matrix_takes_one_launch(cuda, u, kind):
    import torch
    from torch.profiler import ProfilerActivity, profile
    rng = np.random.default_rng(u)
    t = np.ones((u, u), np.float32)
    if kind == "noise":
        t = rng.random((u, u), np.float32)
    else:  # as many minima as there can be, in the corners' cells too
        t[::2, ::2] = 0.25 + 0.5 * rng.random(t[::2, ::2].shape, np.float32)
    d = torch.tensor(t.reshape(-1), device=cuda)
    fip.locate_transients(d, 8 * u, 8, 1e-4, threshold=1.0, max_out=4)  # the block exists
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        got, found = fip.locate_transients(d, 8 * u, 8, 1e-4, threshold=1.0, max_out=u * u)
    launches = sum("LaunchKernel" in e.name for e in p.events())
    want = oracle.locate(t, 8 * u, 8, 1e-4, 1.0)
    if kind == "grid":
        assert len(want) == ((u + 1) // 2) ** 2
    assert found == len(want) == len(got)
    assert [(int(g["tile_row"]), int(g["tile_col"])) for g in got] == [(w[0], w[1]) for w in want]
    assert (got["tlisi"] == np.array([w[2] for w in want], np.float32)).all()
    assert np.abs(got["row"] - [w[3] for w in want]).max() <= 1e-3
    assert np.abs(got["col"] - [w[4] for w in want]).max() <= 1e-3
    assert launches == 1
