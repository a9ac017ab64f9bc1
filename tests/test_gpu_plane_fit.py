"""GPU tests of the plane fit's two forms (one cluster up to 2^16 samples, the
spread form beyond) against an FP64 numpy fit of the same FP32 uvw and
frequencies, at the edges of each form.

Tolerances: V and B are FP64 results rounded once to FP32 (half an ulp, 2^-24
relative); the FP64 fit itself is exact to ~1e-14 over the eigenvalue gap
(>= 0.05 of the trace for these layouts), far below that.
"""
import numpy as np
import pytest

import fastimagingpipe_b200 as fip
from fastimagingpipe_b200 import synthetic

pytestmark = pytest.mark.gpu
C = 299792458.0


def fit64(uvw, freqs):
    k = freqs.astype(np.float64) / C
    x = np.concatenate([uvw.astype(np.float64) * s for s in k])
    B, V = synthetic.plane_fit(x)
    return B, V, np.linalg.norm(x, axis=1)


@pytest.mark.parametrize("rows,chans,offset", [
    (3, 1, 0), (31, 7, 1), (8192, 1, 0), (1128, 3, 2), (130816, 1, 0),
    (32768, 2, 0),                   # 2^16 samples: the last of the one-cluster form
    (32769, 2, 1), (65537, 1, 0),    # the spread form, B off an 8-byte boundary
    (40, 700, 0), (40, 7001, 0), (5, 52500, 1),  # more channels than a CTA stages
    (130816, 8, 0)])
def test_plane_fit_forms(cuda, rows, chans, offset):
    import torch
    rng = np.random.default_rng(rows * 31 + chans)
    # A tilted, flattened cloud away from the origin.
    q, _ = np.linalg.qr(rng.standard_normal((3, 3)))
    uvw = ((rng.standard_normal((rows, 3)) * [900.0, 500.0, 2.0]) @ q.T +
           [40.0, -90.0, 15.0]).astype(np.float32)
    freqs = np.linspace(130e6, 150e6, chans).astype(np.float32)
    ns = rows * chans
    buf = torch.full((2 * ns + 8,), -7.0, device=cuda)
    V = torch.zeros(9, device=cuda)
    fip.plane_project(torch.tensor(uvw.reshape(-1), device=cuda),
                      torch.tensor(freqs, device=cuda), rows, chans,
                      buf.data_ptr() + 4 * offset, V)
    got = buf.cpu().numpy()
    assert (got[:offset] == -7.0).all() and (got[offset + 2 * ns:] == -7.0).all()
    B64, V64, size = fit64(uvw, freqs)
    assert np.abs(V.cpu().numpy().reshape(3, 3) - V64).max() <= 2.0 ** -24 + 1e-9
    err = np.abs(got[offset:offset + 2 * ns].reshape(-1, 2) - B64)
    assert (err <= 2.0 ** -24 * np.abs(B64) + 1e-9 * size[:, None] + 1e-30).all()


def test_single_row_is_the_identity(cuda):
    import torch
    uvw = torch.tensor([3.0, -4.0, 12.0], device=cuda)
    freqs = torch.tensor([140e6], device=cuda)
    B, V = torch.zeros(2, device=cuda), torch.zeros(9, device=cuda)
    fip.plane_project(uvw, freqs, 1, 1, B, V)
    assert np.array_equal(V.cpu().numpy().reshape(3, 3), np.eye(3, dtype=np.float32))
    k = np.float64(np.float32(140e6)) / C
    assert np.allclose(B.cpu().numpy(), [3.0 * k, -4.0 * k], rtol=2.0 ** -23, atol=0)
