"""GPU test of the accuracy of the precision form's steps from the uv grid to the
image -- transform, correction and the reprojection by destination pixel --
against FP64 steps from the same grid, over planes whose curvature lies below and
above the plan's line between its two forms.

The visibilities are noise on baselines up to the grid's edge, so the image
varies by its own RMS from pixel to pixel (its RMS gradient along an axis is
2 pi times the coverage's RMS frequency, 0.16 cycles a pixel: 1.0 a pixel) and
an error of the targets shows in full.  Tolerance: targets off by 1.3e-6 pixel
RMS along each axis move the image by 1.3e-6 x sqrt(2) x 1.0, over the 0.9 that
bilinear weights leave of its amplitude: 2.0e-6; the FP32 transform and
correction add 1e-6 in quadrature (a few 2^-24 per pass): 2.3e-6 relative RMS,
2.5e-6 with a margin.  (Targets off by 2.6e-6 RMS, as with source positions in
the coordinates of a patch of 100 pixels, give 3.3e-6 to 4e-6.)
"""
import numpy as np
import pytest

import fastimagingpipe_b200 as fip
from fastimagingpipe_b200 import synthetic

pytestmark = pytest.mark.gpu


def reproject64(pre, V, cell):
    """The exact map's forward bilinear splat of pre [n, n] in FP64."""
    import torch
    n, h = pre.shape[0], pre.shape[0] // 2
    V = V.double().reshape(3, 3)
    c, a22 = float(np.float32(cell)), abs(float(V[2, 2]))
    off = torch.arange(n, device=pre.device, dtype=torch.float64) - h
    a, b = off[None, :], off[:, None]
    p1 = (-V[0, 0] * a + V[1, 0] * b) / a22
    p2 = (-V[0, 1] * a + V[1, 1] * b) / a22
    rho = c * c * ((p1 - 1) ** 2 + (p2 - 1) ** 2)
    z = torch.where(rho <= 1, rho / (1 + torch.sqrt((1 - rho).clamp(min=0))) / c, 0 * rho)
    ll, mm = p1 - V[2, 0] / V[2, 2] * z, p2 + V[2, 1] / V[2, 2] * z
    ok = (ll.abs() < h - 1) & (mm.abs() < h - 1)
    fl, fm = torch.floor(ll), torch.floor(mm)
    out = torch.zeros(n * n, device=pre.device, dtype=torch.float64)
    for dy, wy in ((0, 1 - mm + fm), (1, mm - fm)):
        for dx, wx in ((0, 1 - ll + fl), (1, ll - fl)):
            at = ((fm + dy + h) * n + fl + dx + h).long()
            out.index_add_(0, at[ok], (pre * wy * wx)[ok])
    return out.reshape(n, n)


def after_grid_error(cuda, n, cell, ha, dec, border=0):
    """Relative RMS error of one snapshot's image against FP64 steps from its own grid, up to
    the taper's constant factor, without `border` pixels along the edges."""
    import torch
    radius = 0.5 / cell * (299792458.0 / 140e6) / 2
    snap = synthetic.make_snapshots(n_ant=60, radius_m=radius, image_size=n, cell_size=cell,
                                    unit_size=4, hour_angle0_h=ha, dec_deg=dec, n_snap=1, seed=n)
    rng = np.random.default_rng(n)
    for k in ("vis_re", "vis_im"):
        getattr(snap, k)[:] = rng.standard_normal(getattr(snap, k).shape)
    nb = snap.num_baselines
    d = [torch.tensor(getattr(snap, k), device=cuda) for k in ("vis_re", "vis_im", "B", "V")]
    img = torch.zeros(n, n, device=cuda)
    with fip.Imager(n, nb, cell, 4, form=fip.FORM_PRECISE) as im:
        im.image_snapshot(*d, nb, img)
        im.check()
        g = im.grid_side
        grid = torch.zeros(g, g // 2 + 1, 2, device=cuda)
        im.grid_snapshot(*d, nb, grid)
        torch.cuda.synchronize()
    sky = torch.fft.irfft2(torch.view_as_complex(grid.double()), s=(g, g), norm="forward")
    at = (torch.arange(n, device=cuda) - n // 2) % g
    # The taper: the transform of exp(beta (sqrt(1 - x^2) - 1)), |x| <= 1, by quadrature.
    x, w = np.polynomial.legendre.leggauss(40)
    w = w * np.exp(15.3704324328 * (np.sqrt(1 - x * x) - 1))
    t = np.cos(np.pi * 8 / g * np.abs(np.arange(n) - n // 2)[:, None] * x) @ w
    t = torch.tensor(t, device=cuda)
    want = reproject64((sky[at][:, at] / (t[:, None] * t[None, :])).abs(), d[3][:9], cell)
    got = img.double()
    if border:
        got, want = (x[border:-border, border:-border] for x in (got, want))
    want = want * float((want * got).sum() / (want * want).sum())
    return float((got - want).square().mean().sqrt() / want.square().mean().sqrt())


@pytest.mark.parametrize("n,cell,ha,dec", [
    (768, 1e-6, 1.5, -30.0), (772, 2e-5, 0.1, -27.0), (1024, 7.3e-6, 1.5, -30.0),
    (1400, 1.4e-5, 1.5, -30.0), (1000, 3e-5, 1.5, -30.0), (1000, 3e-5, 3.0, -30.0),
    (1028, 7.3e-6, 4.0, -10.0), (1028, 1.2e-5, -2.0, -60.0), (900, 3.9e-5, 2.0, -30.0)])
def test_pull_target_accuracy(cuda, n, cell, ha, dec):
    assert after_grid_error(cuda, n, cell, ha, dec) <= 2.5e-6
