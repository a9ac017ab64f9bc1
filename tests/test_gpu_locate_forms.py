"""GPU test of the transient search's two forms against the rule restated in
oracle.locate: identical tiles, tLISI values, order and count; positions to
1e-3 pixel (FP32 centroids of at most 4096 pixels: 2^-12 of a pixel each step).
"""
import numpy as np
import pytest

import fastimagingpipe_b200 as fip
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("u,step", [(1, 0), (33, 3), (256, 5), (256, 2), (512, 16), (513, 16)])
def test_locate_forms(cuda, u, step):
    """One-launch search (up to 2^18 tiles and 4,095 records) and the general
    form: the same tiles, order and count as the restated rule."""
    import torch
    rng = np.random.default_rng(u + step)
    t = np.ones((u, u), np.float32)
    if step:  # isolated minima, some of them equal
        t[::step, ::step] = (0.5 + 0.01 * rng.integers(0, 40, t[::step, ::step].shape)).astype(
            np.float32)
    else:
        t[0, 0] = 0.25
    d = torch.tensor(t.reshape(-1), device=cuda)
    for max_out in (0, 7, u * u):
        got, found = fip.locate_transients(d, 8 * u, 8, 1e-4, threshold=0.95, max_out=max_out)
        want = oracle.locate(t, 8 * u, 8, 1e-4, 0.95)
        assert found == len(want) and len(got) == min(found, max_out)
        for g, w in zip(got, want):
            assert (int(g["tile_row"]), int(g["tile_col"])) == (w[0], w[1])
            assert float(g["tlisi"]) == np.float32(w[2])
            assert abs(float(g["row"]) - w[3]) <= 1e-3 and abs(float(g["col"]) - w[4]) <= 1e-3
