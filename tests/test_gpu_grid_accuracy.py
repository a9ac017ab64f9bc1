"""GPU test of the accuracy of the precision form's uv grid (one and two entries per
thread) against FP64 sums of the same taps, on baselines over the whole grid.

Tolerance: a tap is the product of two values exp(15.4 (sqrt(1 - x^2) - 1)) in
FP32, whose exponents carry the roundings of a square root, a difference and a
product, 2^-24 each (the square root's approximation twice that), times 15.4: 1e-6
relative RMS, 1.4e-6 for the two factors; the distance of a tap, one rounding of a
few cells (2^-23 cell), adds 1e-7 and the sums 1e-7.  2.5e-6 leaves the rest to
spare.  (Distances from positions rounded to FP32 first, half an ulp of hundreds of
cells, give 5e-6 to 1e-5.)
"""
import numpy as np
import pytest

import fastimagingpipe_b200 as fip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nb", [(772, 3000), (1024, 1500), (1400, 200000)])
def test_grid_matches_fp64(cuda, n, nb):
    import torch
    cell = 0.02 / n
    rng = np.random.default_rng(n)
    lim = 0.47 / cell  # wavelengths: no tap beyond the grid's edge
    B = rng.uniform(-lim, lim, (nb, 2)).astype(np.float32)
    vis = rng.standard_normal((2, nb)).astype(np.float32)
    V = np.array([0.9, 0.1, 0.4, -0.2, 0.95, 0.2, -0.37, -0.26, 0.88], np.float32)
    d = [torch.tensor(x, device=cuda) for x in (vis[0], vis[1], B.reshape(-1), V)]
    with fip.Imager(n, nb, cell, 4, form=fip.FORM_PRECISE) as im:
        g = im.grid_side
        grid = torch.zeros(g, g // 2 + 1, 2, device=cuda)
        im.grid_snapshot(*d, nb, grid)
        torch.cuda.synchronize()
    scale = float(np.float32(cell) * np.float32(g))
    inten = abs(float(V[0]) * float(V[4]) - float(V[1]) * float(V[3]))
    beta = float(np.float32(15.3704324328))
    p = torch.tensor(B, device=cuda).double() * scale
    w = torch.complex(d[0].double(), d[1].double()) / inten
    lo = torch.ceil(p - 4)
    full = torch.zeros(g * g, dtype=torch.complex128, device=cuda)
    es = lambda x: torch.where(x.abs() <= 1, torch.exp(
        beta * (torch.sqrt((1 - x * x).clamp(min=0)) - 1)), torch.zeros_like(x))
    for a in range(9):
        for b in range(9):
            r = lo + torch.tensor([a, b], device=cuda, dtype=torch.float64)
            k = es((r[:, 0] - p[:, 0]) / 4) * es((r[:, 1] - p[:, 1]) / 4)
            at = (r[:, 0].long() % g) * g + r[:, 1].long() % g
            full.index_add_(0, at, w * k)
    full = full.reshape(g, g)
    i = (-torch.arange(g, device=cuda)) % g
    want = (0.5 * (full + full[i][:, i].conj()))[:, :g // 2 + 1]
    got = torch.view_as_complex(grid.double())
    err = float((got - want).abs().square().mean().sqrt() / want.abs().square().mean().sqrt())
    assert err <= 2.5e-6
