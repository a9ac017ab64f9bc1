"""GPU test of the tile binning at its edges, through the gridding entry points:
grids of one, two and many tiles, footprints that wrap and that reach past
the grid, counts around a CTA's share, unaligned coordinates, positions
without a footprint (NaN, infinite, far outside).

The grid is compared with a plain FP64 restatement of the definition in
include/fip.h (fip_grid_snapshot).  Tolerance: the plain form's sums are FP32
taps in fixed point of 2^-30 of a work item's summed weights: 2e-6 of the
grid's largest cell covers both.
"""
import numpy as np
import pytest

import fastimagingpipe_b200 as fip

pytestmark = pytest.mark.gpu
BETA = 15.3704324328


def grid64(vr, vi, B, V, n, cell):
    g = int(np.ceil(1.5 * n))
    sc = np.float32(cell) * np.float32(g)
    w = (vr.astype(np.float64) + 1j * vi) / abs(float(V[0]) * V[4] - float(V[1]) * V[3])
    full = np.zeros((g, g), np.complex128)
    tap = np.arange(9)
    for k, (p1, p2) in enumerate((B * sc).astype(np.float32).astype(np.float64)):
        if not (abs(p1) < 1e9 and abs(p2) < 1e9):
            continue
        r = [np.ceil(p - 4).astype(int) + tap for p in (p1, p2)]
        ker = []
        for rr, p in zip(r, (p1, p2)):
            x = (rr - p) / 4
            ok = (np.abs(x) <= 1) & (rr >= -(g // 2)) & (rr <= (g - 1) // 2)
            ker.append(np.where(ok, np.exp(BETA * (np.sqrt(np.maximum(1 - x * x, 0)) - 1)), 0))
        np.add.at(full, (r[0][:, None] % g, r[1][None, :] % g), w[k] * np.outer(*ker))
    neg = np.roll(np.roll(full[::-1, ::-1], 1, 0), 1, 1)
    return ((full + neg.conj()) / 2)[:, :g // 2 + 1]


@pytest.mark.parametrize("n", [16, 40, 44, 48, 100, 256, 1000])
@pytest.mark.parametrize("nb,offset", [(1, 0), (511, 1), (2048, 0), (5000, 1)])
def test_binned_grid(cuda, n, nb, offset):
    import torch
    rng = np.random.default_rng(n * 7 + nb)
    cell, g = 1e-4, int(np.ceil(1.5 * n))
    half = g / 2
    p = rng.uniform(-half - 3, half + 3, (nb, 2))
    core = rng.random(nb) < 0.4  # a dense core: tiles split over work items
    p[core] = rng.uniform(-6, 6, (int(core.sum()), 2))
    edge = rng.random(nb) < 0.1
    p[edge, 1] = rng.choice([-half, 0.0, half - 1, -0.5], int(edge.sum()))
    B = (p / (cell * g)).astype(np.float32)
    bad = rng.random(nb) < 0.02
    B[bad, 0] = rng.choice([np.nan, np.inf, -1e30, 1e9], int(bad.sum()))
    vr, vi = rng.standard_normal((2, nb)).astype(np.float32)
    V = np.linalg.qr(rng.standard_normal((3, 3)))[0].astype(np.float32).reshape(-1)
    dev = lambda a: torch.tensor(np.ascontiguousarray(a), device=cuda)
    buf = torch.zeros(2 * nb + 4, device=cuda)
    buf[offset:offset + 2 * nb] = dev(B.reshape(-1))
    d = dict(vr=dev(vr), vi=dev(vi), V=dev(V))
    want = grid64(vr, vi, B, V, n, cell)
    tol = 2e-6 * max(float(np.abs(want).max()), 1e-30)
    out = torch.full((g, g // 2 + 1, 2), 3.0, device=cuda)
    with fip.Imager(n, nb, cell, 0) as im:
        for _ in range(2):  # the second call on used scratch
            im.grid_snapshot(d["vr"], d["vi"], buf.data_ptr() + 4 * offset, d["V"], nb, out)
    free = torch.full((g, g // 2 + 1, 2), 3.0, device=cuda)
    fip.grid_snapshot_noalloc(d["vr"], d["vi"], buf.data_ptr() + 4 * offset, d["V"], nb, n, cell,
                              free)
    for got in (out, free):
        got = got.cpu().numpy().astype(np.float64)
        assert np.abs(got[..., 0] + 1j * got[..., 1] - want).max() <= tol
