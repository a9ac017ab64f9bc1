"""GPU test of the plane fit of few rows and many channels: the values against
an FP64 fit, at the edges of the two ways to sum the channels (up to 256 by one
warp) and to spread the samples, beyond 65,535 blocks of 256 channels, and the
time against a fit of as many samples in one channel.

Tolerances: V and B are FP64 results rounded once to FP32 (half an ulp, 2^-24
relative); the fit itself is exact to ~1e-13 over the eigenvalue gap (>= 0.05 of
the trace for these layouts), far below 1e-9.
"""
import numpy as np
import pytest

import fastimagingpipe_b200 as fip

pytestmark = pytest.mark.gpu
C = 299792458.0


def layout(rows, seed):
    """A tilted, flattened cloud away from the origin, well spread for any number of rows."""
    rng = np.random.default_rng(seed)
    q, _ = np.linalg.qr(rng.standard_normal((3, 3)))
    a = 2 * np.pi * np.arange(rows) / rows + 0.3
    p = np.stack([900 * np.cos(a), 500 * np.sin(a), 2 * rng.standard_normal(rows)], 1)
    return (p @ q.T + [40.0, -90.0, 15.0]).astype(np.float32)


@pytest.mark.parametrize("rows,chans,offset", [
    (3, 256, 0), (3, 257, 1), (1, 65536, 0), (5, 13107, 0), (2047, 31, 0), (2048, 32, 0),
    (2047, 33, 0), (255, 300, 1), (256, 300, 0), (1, 65537, 0), (4, 400001, 0),
    (2, 65535 * 256 + 1, 0)])
def test_values(cuda, rows, chans, offset):
    import torch
    uvw = layout(rows, rows + chans)
    freqs = np.linspace(130e6, 150e6, chans).astype(np.float32)
    ns = rows * chans
    buf = torch.full((2 * ns + 8,), -7.0, device=cuda)
    V = torch.zeros(9, device=cuda)
    fip.plane_project(torch.tensor(uvw.reshape(-1), device=cuda),
                      torch.tensor(freqs, device=cuda), rows, chans,
                      buf.data_ptr() + 4 * offset, V)
    # The FP64 fit, its sums factored over rows and channels.
    u, k = uvw.astype(np.float64), freqs.astype(np.float64) / C
    m = u.mean(0)
    cov = (k ** 2).sum() * ((u - m).T @ (u - m)) + rows * ((k - k.mean()) ** 2).sum() * np.outer(
        m, m)
    _, q = np.linalg.eigh(cov / np.trace(cov))
    ax = [q[:, 2], q[:, 1]]
    ax = [a * np.sign(a[np.argmax(np.abs(a))]) for a in ax]
    V64 = np.stack(ax + [np.cross(ax[0], ax[1])])
    got_v = V.cpu().numpy().reshape(3, 3)
    axes = 2 if rows > 1 else 1  # one row: the second axis is any normal of the first
    assert np.abs(got_v[:axes] - V64[:axes]).max() <= 2.0 ** -24 + 1e-9
    got = buf[offset:offset + 2 * ns].view(chans, rows, 2)
    dk = torch.tensor(k, device=cuda)[:, None]
    size = torch.tensor(np.linalg.norm(u, axis=1), device=cuda)[None] * dk
    for a in range(2):
        want = torch.tensor(u @ V64[a] if a < axes else np.zeros(rows), device=cuda)[None] * dk
        err = (got[:, :, a].double() - want).abs() - 2.0 ** -24 * want.abs() - 1e-9 * size
        assert float(err.max()) <= 0
    assert bool((buf[:offset] == -7.0).all()) and bool((buf[offset + 2 * ns:] == -7.0).all())


@pytest.mark.parametrize("rows,chans", [(1, 65536), (5, 13107), (5, 52500), (1, 1 << 20)])
def test_many_channels_take_the_time_of_as_many_rows(cuda, rows, chans):
    """Both fit and write the same number of samples; the channels add a division
    each and the rows a load of their coordinates, so neither takes four times
    the other's time (a fit that leaves the channels to few threads: thirty)."""
    import torch

    def best_us(r, c):
        uvw = torch.randn(3 * r, device=cuda)
        freqs = torch.linspace(130e6, 150e6, c, device=cuda)
        B, V = torch.zeros(2 * r * c, device=cuda), torch.zeros(9, device=cuda)
        times = []
        for _ in range(20):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            a.record()
            for _ in range(5):
                fip.plane_project(uvw, freqs, r, c, B, V)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return 200 * min(times)

    assert best_us(rows, chans) <= 4 * best_us(rows * chans, 1)
