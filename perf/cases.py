"""The work that users of this framework have it do, as measurable cases.

Every case goes through public entry points only: the drop-in call on host
buffers (FIpipe), three-snapshot calls on device buffers (Imager.pipe_device),
one beam's run of snapshots (Imager.image_sequence), mixed-size and
multi-channel batches (Batch), raw samples with the device plane fit and the
Stokes-I collapse, the sliding-window trigger followed by the transient
search, and the multi-beam server.  Inputs are seeded synthetic snapshots of
an Earth-rotating array (the layouts, sky and noise of the benchmark
configurations), made on the GPU.

A case is a dict: "op" (the entry point), "n" (image side), "antennas" and
"chans" (samples per snapshot = antennas (antennas - 1) / 2 * chans),
"radius" (array radius in metres), "cell" (radians per pixel), "tile"
(trigger tile), "snaps" (snapshots per pass), "form" (plain, or the precision
form by visibility storage: f32, f16, bf16), "flagged" (the largest share of
a snapshot's samples flagged), and for two-size work "n2", the second image
side (its cell scaled to the same field of view).
"""
import math

import numpy as np
import torch

import fastimagingpipe_b200 as fip

C_LIGHT = 299792458.0
ES_BETA, ES_NORM = 15.3704324328, 2.4937047051153827  # the gridding kernel's constants
DEV = "cuda:0"
BIG_CELL = 7.2722e-6  # radians per pixel of the 4096 x 4096 field


def _case(name, op, n, antennas, form, **kw):
    c = dict(name=name, op=op, n=n, n2=0, antennas=antennas, chans=1, radius=20000.0,
             cell=BIG_CELL * 4096 / n, tile=32, snaps=3, form=form, flagged=0.0)
    c.update(kw)
    return c


def listed():
    return [
        # The drop-in call of a program written for the reference: host
        # buffers in, tLISI matrix out, the benchmark's shape.
        _case("fipipe_host_4096", "pipe_host", 4096, 512, "plain"),
        # The same three snapshots resident in HBM, reference-faithful form.
        _case("pipe_plain_4096", "pipe", 4096, 512, "plain"),
        # ... and the precision form with half-width visibility storage.
        _case("pipe_f16_4096", "pipe", 4096, 512, "f16"),
        # A small array's monitor: 128 antennas on 512 x 512, where launches
        # and latency count.
        _case("pipe_plain_512", "pipe", 512, 128, "plain", radius=1000.0, cell=2.9e-5, tile=16),
        # The smallest call: a quick-look image of a 48-antenna array in the
        # precision form.
        _case("pipe_f32_128", "pipe", 128, 48, "f32", radius=1000.0, cell=1.2e-4, tile=16),
        # One beam's run of snapshots on a round decimal image side, uneven
        # counts after flagging.
        _case("sequence_f32_1000", "sequence", 1000, 256, "f32", radius=5000.0, tile=20,
              snaps=10, flagged=0.2),
        # One snapshot at a large side that is not a power of two: plane fit,
        # collapse, image, as separate calls.
        _case("snapshot_plain_3000", "snapshot", 3000, 512, "plain", radius=14000.0, tile=24,
              snaps=1, flagged=0.1),
        # Multi-frequency batches of two image sizes, up to 30 % flagged.
        _case("batch_plain_mixed", "batch", 4096, 512, "plain", n2=2048, chans=8, snaps=4,
              flagged=0.3),
        # The precision form's batches of one size, wider uv coverage.
        _case("batch_bf16_2048", "batch", 2048, 512, "bf16", chans=4, snaps=8, flagged=0.3),
        # Raw two-polarisation samples of one snapshot: plane fit on the
        # device, then the collapse inside the gridder's load.
        _case("ingest_plain_2048", "ingest", 2048, 512, "plain", chans=8, radius=10000.0,
              snaps=1, flagged=0.2),
        # The trigger over a run of images and the search of every tLISI
        # matrix for transients.
        _case("window_plain_4096", "window", 4096, 48, "plain", snaps=8),
        # A server with beams of two sizes, a burst of requests.
        _case("serve_plain_2048", "serve", 2048, 512, "plain", n2=1024, snaps=4, radius=10000.0),
    ]


def draw(rng):
    """One more case of the same ranges: sides 128 .. 4096 in steps of four (spread over
    their logarithm), powers of two half of the time, 48 .. 512 antennas to match."""
    def side(lo, hi):
        v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        if rng.random() < 0.5:
            return min(1 << round(math.log2(v)), hi)
        return max(lo, min(hi, 4 * round(v / 4)))

    op = rng.choice(["pipe_host", "pipe", "pipe", "pipe", "sequence", "snapshot", "batch",
                     "ingest", "window", "serve"])
    n = side(128, 4096)
    if op in ("serve", "batch"):
        n = side(256, 2048)
    frac = math.log2(n / 128) / 5  # 0 .. 1 over the range
    antennas = rng.randint(48, 96 + int(416 * frac))
    form = "plain" if op in ("pipe_host", "window") else rng.choice(
        ["plain", "plain", "f32", "f16", "bf16"])
    # Baselines up to between a tenth and half of the grid's half side.
    cell = BIG_CELL * 4096 / n * rng.uniform(0.8, 1.3)
    reach = rng.uniform(0.1, 0.5) * 0.5 / cell  # wavelengths
    radius = reach * C_LIGHT / 140e6 / 2
    tile = rng.choice([t for t in (8, 16, 20, 24, 32) if t <= n // 4])
    chans = rng.choice([1, 1, 2, 4]) if op in ("batch", "ingest", "snapshot") else 1
    snaps = {"pipe": 3, "pipe_host": 3, "sequence": rng.randint(4, 8), "snapshot": 1,
             "batch": rng.randint(2, 6), "ingest": 1, "window": rng.randint(4, 8),
             "serve": rng.randint(2, 4)}[op]
    n2 = 0
    if op == "serve" or (op == "batch" and rng.random() < 0.5):
        n2 = side(128, n)
    flagged = 0.0 if op in ("pipe", "pipe_host", "window", "serve") else rng.uniform(0.0, 0.3)
    c = _case("", op, n, antennas, form, n2=n2, chans=chans, radius=radius, cell=cell,
              tile=tile, snaps=snaps, flagged=flagged)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _kw(form):
    if form == "plain":
        return {}
    return dict(form=fip.FORM_PRECISE,
                vis_storage={"f32": fip.STORE_F32, "f16": fip.STORE_F16,
                             "bf16": fip.STORE_BF16}[form])


def _sizes(case):
    """(n, cell) of each of the case's image sizes."""
    out = [(case["n"], case["cell"])]
    if case["n2"]:
        out.append((case["n2"], case["cell"] * case["n"] / case["n2"]))
    return out


def _baselines(case, g):
    """Equatorial baseline vectors in metres [nb, 3], FP64: half of the antennas uniform in
    the array's disk, half in a core a twentieth as wide."""
    na = case["antennas"]
    rad = torch.sqrt(torch.rand(na, generator=g, device=DEV, dtype=torch.float64))
    rad = rad * case["radius"] * torch.where(torch.arange(na, device=DEV) < na // 2, 0.05, 1.0)
    th = 2 * math.pi * torch.rand(na, generator=g, device=DEV, dtype=torch.float64)
    lat = math.radians(-26.7)
    e, nn = rad * torch.cos(th), rad * torch.sin(th)
    xyz = torch.stack([-math.sin(lat) * nn, e, math.cos(lat) * nn], 1)
    i, j = torch.triu_indices(na, na, 1, device=DEV)
    return xyz[j] - xyz[i]


def _uvw(xyz, k):
    """uvw in metres of snapshot k, ten seconds apart, declination -30 degrees."""
    ha = 2 * math.pi * (1.5 * 3600 + 10.0 * k) / 86164.0905
    sh, ch, sd, cd = math.sin(ha), math.cos(ha), math.sin(math.radians(-30)), math.cos(
        math.radians(-30))
    x, y, z = xyz.unbind(1)
    return torch.stack([sh * x + ch * y, -sd * ch * x + sd * sh * y + cd * z,
                        cd * ch * x - cd * sh * y + sd * z], 1)


def _plane_fit(x):
    """FP64 plane fit of uvw in wavelengths: (B [nb, 2], V [3, 3]).  Rows 0 and 1 of V are the
    first two principal axes, their largest components positive."""
    xc = x - x.mean(0)
    _, q = np.linalg.eigh((xc.T @ xc).cpu().numpy())
    v = np.stack([q[:, 2], q[:, 1]])
    for r in range(2):
        if v[r, np.argmax(np.abs(v[r]))] < 0:
            v[r] = -v[r]
    v = np.concatenate([v, np.cross(v[0], v[1])[None]])
    return x @ torch.tensor(v[:2].T.copy(), device=DEV), torch.tensor(v, device=DEV)


def _freqs(case):
    f = [140e6] if case["chans"] == 1 else list(np.linspace(130e6, 150e6, case["chans"]))
    return torch.tensor(f, device=DEV, dtype=torch.float32)


def _snapshots(case, seed, n, cell, sub=0):
    """The case's snapshots for one image size: dicts of device tensors.  vis, B and V for the
    calls that take visibilities, the raw samples (xx, yy, flags, weights) and uvw for those
    that take them."""
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 31 * sub + 1)
    r = lambda *s: torch.rand(*s, generator=g, device=DEV, dtype=torch.float64)
    rn = lambda *s: torch.randn(*s, generator=g, device=DEV, dtype=torch.float64)
    xyz = _baselines(case, g)
    half = 0.2 * n * cell
    src = torch.cat([2 * half * (r(20, 2) - 0.5), torch.exp(rn(20, 1))], 1)
    trans = torch.cat([2 * half * (r(1, 2) - 0.5), torch.full((1, 1), 5.0, device=DEV,
                                                               dtype=torch.float64)], 1)
    freqs = _freqs(case)
    raw = case["op"] in ("snapshot", "ingest")
    out = []
    for k in range(case["snaps"]):
        uvw = _uvw(xyz, k).float()
        x = torch.cat([uvw.double() * (float(f) / C_LIGHT) for f in freqs])
        sky = src if k != case["snaps"] - 1 else torch.cat([src, trans])
        vis = torch.zeros(x.shape[0], device=DEV, dtype=torch.complex128)
        for l, m, flux in sky.tolist():
            ph = x[:, 0] * l + x[:, 1] * m + x[:, 2] * (math.sqrt(1 - l * l - m * m) - 1)
            ph = -2 * math.pi * (ph - torch.round(ph))
            vis += flux * torch.complex(torch.cos(ph), torch.sin(ph))
        d = {}
        if raw:
            q = 0.3 * vis.abs() * torch.complex(rn(x.shape[0]), rn(x.shape[0]))
            for pol, sign in ((0, 1), (3, -1)):
                v = vis + sign * q + 0.1 * torch.complex(rn(x.shape[0]), rn(x.shape[0]))
                d["re%d" % pol] = v.real.float().contiguous()
                d["im%d" % pol] = v.imag.float().contiguous()
                d["flag%d" % pol] = (r(x.shape[0]) < case["flagged"]).to(torch.uint8)
                d["weight%d" % pol] = (0.5 + r(x.shape[0])).float()
            d["uvw"], d["nb"] = uvw.contiguous(), x.shape[0]
        else:
            vis = vis + 0.1 * torch.complex(rn(x.shape[0]), rn(x.shape[0]))
            b, v = _plane_fit(x)
            if case["flagged"]:
                keep = r(x.shape[0]) >= case["flagged"] * float(r(1))
                vis, b = vis[keep], b[keep]
            d = dict(re=vis.real.float().contiguous(), im=vis.imag.float().contiguous(),
                     B=b.float().reshape(-1).contiguous(), V=v.float().reshape(-1).contiguous(),
                     nb=int(vis.numel()))
        out.append(d)
    return out


def _images(case, seed):
    """A run of positive images as the imager leaves them: a noise floor, steady sources as
    wide as the beam, small changes between snapshots, a transient in the middle one."""
    n, s = case["n"], case["snaps"]
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 17)
    base = torch.randn(n, n, generator=g, device=DEV).abs_()
    at = torch.randint(8, n - 8, (21, 2), generator=g, device=DEV).tolist()
    flux = torch.exp(torch.randn(21, generator=g, device=DEV)).mul_(20).tolist()
    d = torch.arange(-8, 8, device=DEV, dtype=torch.float32)
    beam = torch.exp(-(d[:, None] ** 2 + d[None, :] ** 2) / 8)
    for (y, x), f in zip(at[:20], flux[:20]):
        base[y - 8:y + 8, x - 8:x + 8] += f * beam
    imgs = torch.empty(s, n, n, device=DEV)
    for k in range(s):
        torch.randn(n, n, generator=g, device=DEV, out=imgs[k])
        imgs[k].mul_(0.1).add_(base).abs_()
        if k == s // 2:
            y, x = at[20]
            imgs[k][y - 8:y + 8, x - 8:x + 8] += 150 * beam
    return imgs, imgs.reshape(s, -1).max(dim=1).values.contiguous()


class _DeviceView:
    """A device buffer owned by an imager, for torch.as_tensor; keeps its owner alive."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f4", data=(ptr, False),
                                             version=3)


def _host(snaps, key):
    return torch.cat([s[key] for s in snaps]).cpu().numpy()


def prepare(case, seed):
    op, n, cell, t, kw = case["op"], case["n"], case["cell"], case["tile"], _kw(case["form"])
    u = n // t
    st = dict(op=op, case=case)
    if op == "window":
        st["images"], st["maxima"] = _images(case, seed)
        st["out"] = torch.zeros(case["snaps"] - 2, u, u, device=DEV)
        st["im"] = fip.Imager(n, 16, cell, t, **kw)
        return st
    groups = [_snapshots(case, seed, nn, cc, k) for k, (nn, cc) in enumerate(_sizes(case))]
    snaps = groups[0]
    nbmax = max(s["nb"] for q in groups for s in q)
    if op == "pipe_host":
        st["args"] = tuple(_host(snaps, k) for k in ("re", "im", "B", "V"))
        st["nb"] = nbmax
    elif op == "pipe":
        st["args"] = tuple(torch.cat([s[k] for s in snaps]) for k in ("re", "im", "B", "V"))
        st["nb"] = nbmax
        st["out"] = torch.zeros(u, u, device=DEV)
        st["im"] = fip.Imager(n, nbmax, cell, t, **kw)
        st["images"] = [torch.as_tensor(_DeviceView(st["im"], st["im"].image_ptr(k), (n, n)),
                                        device=DEV) for k in range(3)]
    elif op == "sequence":
        pad = lambda v, w: torch.nn.functional.pad(v, (0, w * nbmax - v.numel()))
        st["args"] = tuple(torch.cat([pad(s[k], w) for s in snaps])
                           for k, w in (("re", 1), ("im", 1), ("B", 2)))
        st["args"] += (torch.cat([s["V"] for s in snaps]),)
        st["nb"], st["stride"] = [s["nb"] for s in snaps], nbmax
        st["out"] = torch.zeros(case["snaps"] - 2, u, u, device=DEV)
        st["im"] = fip.Imager(n, nbmax, cell, t, **kw)
    elif op in ("snapshot", "ingest"):
        st["snap"], st["freqs"], st["nb"] = snaps[0], _freqs(case), nbmax
        st["B"] = torch.zeros(nbmax, 2, device=DEV)
        st["V"] = torch.zeros(3, 3, device=DEV)
        st["vis"] = torch.zeros(2, nbmax, device=DEV)
        st["image"] = torch.zeros(n, n, device=DEV)
        st["max"] = torch.zeros(1, device=DEV)
        st["im"] = fip.Imager(n, nbmax, cell, t, **kw)
    elif op == "batch":
        flat = [(c, s) for k in range(case["snaps"]) for c, s in
                ((c, q[k]) for c, q in enumerate(groups))]
        st["seq"] = [c for c, _ in flat]
        st["args"] = tuple([s[k] for _, s in flat] for k in ("re", "im", "B", "V", "nb"))
        st["batch"] = fip.Batch.of_sequences([(nn, nbmax, cc, t) for nn, cc in _sizes(case)],
                                             case["snaps"], **kw)
        st["out"] = [torch.zeros(case["snaps"], nn // t, nn // t, device=DEV)
                     for nn, _ in _sizes(case)]
        # The stream runs on: every snapshot of a pass has its predecessors.
        st["batch"].image_sequences(st["seq"], *st["args"], st["out"])
    elif op == "serve":
        st["sv"] = fip.Server(24 << 30, slots=2)
        st["beams"] = [st["sv"].add_beam(nn, nbmax, cc, t, **kw) for nn, cc in _sizes(case)]
        st["req"] = [(b, tuple(q[k][x].cpu().numpy() for x in ("re", "im", "B", "V")), q[k]["nb"])
                     for k in range(case["snaps"]) for b, q in zip(st["beams"], groups)]
        ids = [st["sv"].submit(b, *a, nb) for b, a, nb in st["req"]]
        for i in ids:
            st["sv"].wait(i)
    torch.cuda.synchronize()
    return st


def run(st):
    op, case = st["op"], st["case"]
    if op == "pipe_host":
        return fip.FIpipe(*st["args"], st["nb"], case["n"], 3, case["cell"], case["tile"])
    if op == "pipe":
        st["im"].pipe_device(*st["args"], st["nb"], st["out"])
        return [st["out"]] + st["images"]
    if op == "sequence":
        st["im"].image_sequence(*st["args"], st["nb"], st["stride"], st["out"])
        return st["out"]
    if op in ("snapshot", "ingest"):
        s, chans = st["snap"], case["chans"]
        fip.plane_project(s["uvw"], st["freqs"], s["nb"] // chans, chans, st["B"], st["V"])
        pols = (s["re0"], s["im0"], s["re3"], s["im3"], s["flag0"], s["flag3"], s["weight0"],
                s["weight3"])
        if op == "snapshot":
            fip.collapse_visibilities(*pols, st["vis"][0], st["vis"][1], s["nb"])
            st["im"].image_snapshot(st["vis"][0], st["vis"][1], st["B"], st["V"], s["nb"],
                                    st["image"], st["max"])
            return dict(B=st["B"], V=st["V"], vis=st["vis"], image=st["image"], max=st["max"])
        st["im"].image_snapshot_raw(*pols, st["B"], st["V"], s["nb"], st["image"], st["max"])
        return dict(B=st["B"], V=st["V"], image=st["image"], max=st["max"])
    if op == "batch":
        st["batch"].image_sequences(st["seq"], *st["args"], st["out"])
        return st["out"]
    if op == "window":
        st["im"].trigger_window(st["images"], st["maxima"], case["snaps"], st["out"])
        found = np.zeros(case["snaps"] - 2, np.int64)
        places = np.zeros((case["snaps"] - 2, 64, 7), np.float32)  # fip.LOCATION_DTYPE's fields
        for k in range(case["snaps"] - 2):
            rec, found[k] = fip.locate_transients(st["out"][k], case["n"], case["tile"],
                                                  case["cell"], max_out=64)
            for f, name in enumerate(rec.dtype.names):
                places[k, :len(rec), f] = rec[name]
        return [st["out"], found, places]
    ids = [st["sv"].submit(b, *a, nb) for b, a, nb in st["req"]]
    return [st["sv"].wait(i)["tlisi"] for i in ids]


# ---------------------------------------------------------------------------
# Work and 64-bit values
# ---------------------------------------------------------------------------

def work(case):
    nb = case["antennas"] * (case["antennas"] - 1) // 2 * case["chans"]
    op, s = case["op"], case["snaps"]
    b = f = 0.0
    for n, _ in _sizes(case):
        u, g = n // case["tile"], 1.5 * n
        if op == "window":
            b += 4.0 * s * n * n + 4.0 * (s - 2) * u * u
            f += 10.0 * (s - 2) * n * n
            continue
        kept = 1 - case["flagged"] / 2 if op in ("sequence", "batch") else 1.0
        vis = nb * kept
        # Gridding: a complex multiply-add per tap of 8 x 8; the transform:
        # row pairs of length 1.5 n, half as much for the occupied columns;
        # 60 operations per pixel of mapping and splat, 10 of the trigger.
        f += s * (64 * 4 * vis + 1.5 * (n / 2) * 5 * g * math.log2(g) + 70.0 * n * n)
        b += s * 16.0 * vis
        if op in ("snapshot", "ingest"):
            b += 10.0 * nb + (8.0 * nb if op == "snapshot" else 0.0) + 12.0 * nb / case["chans"]
        if op in ("pipe", "snapshot", "ingest"):
            b += 4.0 * s * n * n  # the images come back
        if op not in ("snapshot", "ingest"):
            b += 4.0 * u * u * (1 if op in ("pipe", "pipe_host") else s)
    return {"bytes": b, "flops": f}


def _taper64(n, g):
    """Grid correction at 0 .. n / 2: the kernel's Fourier integral by 28-node Gauss-Legendre
    quadrature, which defines it."""
    x, w = np.polynomial.legendre.leggauss(28)
    x, w = x[14:], w[14:]
    phi = np.exp(ES_BETA * (np.sqrt(1 - x * x) - 1))
    t = np.arange(n // 2 + 1) / g
    return torch.tensor(8 / ES_NORM * (np.cos(8 * np.pi * t[:, None] * x) @ (phi * w)),
                        device=DEV)


def _image64(re, im, b, v, nb, n, cell):
    """One snapshot's image in 64 bits: gridding, transform, correction, closed-form
    reprojection."""
    g = int(math.ceil(1.5 * n))
    cell = float(np.float32(cell))
    v = v.double().reshape(9).tolist()
    w = torch.complex(re.double(), im.double()) / abs(v[0] * v[4] - v[1] * v[3])
    p = b.double().reshape(-1, 2) * (cell * g)
    grid = torch.zeros(g * g, 2, device=DEV, dtype=torch.float64)
    tap = torch.arange(9, device=DEV)
    for a in range(0, int(w.numel()), 1 << 17):
        q = p[a:a + (1 << 17)]
        r = torch.ceil(q - 4).long()[:, :, None] + tap  # [nb, 2, 9]
        x = (r - q[:, :, None]) / 4
        k = torch.where((x.abs() <= 1) & (r >= -(g // 2)) & (r <= (g - 1) // 2),
                        torch.exp(ES_BETA * (torch.sqrt((1 - x * x).clamp(min=0)) - 1)), 0.0)
        at = ((r[:, 0] % g) * g)[:, :, None] + (r[:, 1] % g)[:, None, :]
        val = torch.view_as_real(w[a:a + (1 << 17)])[:, None, None, :] * (
            k[:, 0, :, None] * k[:, 1, None, :])[..., None]
        grid.index_add_(0, at.reshape(-1), val.reshape(-1, 2))
    full = torch.fft.ifft2(torch.view_as_complex(grid).reshape(g, g), norm="forward").real
    del grid
    h = n // 2
    off = torch.arange(-h, n - h, device=DEV)
    ck = _taper64(n, g)[off.abs()] * ES_NORM
    pre = (full[off % g][:, off % g] / (ck[:, None] * ck[None, :])).abs() / nb
    del full
    i, j = off.double()[None, :], off.double()[:, None]
    a22 = abs(v[8])
    p1, p2 = (-v[0] * i + v[3] * j) / a22, (-v[1] * i + v[4] * j) / a22
    rho = cell * cell * ((p1 - 1) ** 2 + (p2 - 1) ** 2)
    z = torch.where(rho <= 1, rho / (1 + torch.sqrt((1 - rho).clamp(min=0))), 0.0) / cell
    ll, mm = p1 - v[6] / v[8] * z, p2 + v[7] / v[8] * z
    ok = (ll.abs() < h - 1) & (mm.abs() < h - 1)
    ll, mm, pre = ll[ok], mm[ok], pre[ok]
    fl, fm = torch.floor(ll), torch.floor(mm)
    out = torch.zeros(n * n, device=DEV, dtype=torch.float64)
    for dm in (0, 1):
        for dl in (0, 1):
            wt = (ll - fl if dl else 1 - ll + fl) * (mm - fm if dm else 1 - mm + fm)
            out.index_add_(0, ((fm.long() + dm + h) * n + fl.long() + dl + h), wt * pre)
    return out.reshape(n, n)


def _tlisi64(i1, i2, i3, t):
    n = i1.shape[0]
    u = n // t
    d = ((i1 - i2).abs() - (i2 - i3).abs()).abs()
    q = torch.where(i2 <= 0, torch.tensor(1e-6, device=DEV, dtype=torch.float64), i2)
    q = (d / q).clamp(max=1.0)
    tiles = lambda x: x[:u * t, :u * t].reshape(u, t, u, t).permute(0, 2, 1, 3).reshape(u, u, -1)
    mx = max(float(x.max()) for x in (i1, i2, i3))
    d, q = tiles(d), tiles(q)
    return 1 - d.mean(-1) * d.max(-1).values * q.mean(-1) / mx / mx


def exact(case, seed):
    op, t = case["op"], case["tile"]
    if op == "window":
        imgs, _ = _images(case, seed)
        return [torch.stack([_tlisi64(*(imgs[k + j].double() for j in range(3)), t)
                             for k in range(case["snaps"] - 2)]), None, None]
    groups = [(nn, cc, _snapshots(case, seed, nn, cc, k))
              for k, (nn, cc) in enumerate(_sizes(case))]
    if op in ("snapshot", "ingest"):
        n, cell, (s,) = groups[0]
        x = torch.cat([s["uvw"].double() * (float(f) / C_LIGHT) for f in _freqs(case)])
        b, v = _plane_fit(x)
        w0, w3 = (torch.where(s["flag%d" % k] > 0, 0.0, s["weight%d" % k].double())
                  for k in (0, 3))
        ws = w0 + w3
        re, im = (torch.where(ws > 0, (s[c + "0"].double() * w0 + s[c + "3"].double() * w3) /
                              torch.where(ws > 0, ws, 1.0), 0.0) for c in ("re", "im"))
        img = _image64(re, im, b, v, s["nb"], n, cell)
        out = dict(B=b, V=v, image=img, max=img.max().reshape(1))
        if op == "snapshot":
            out["vis"] = torch.stack([re, im])
        return out
    every = []
    for n, cell, snaps in groups:
        imgs = [_image64(s["re"], s["im"], s["B"], s["V"], s["nb"], n, cell) for s in snaps]
        if op in ("pipe", "pipe_host", "sequence"):
            m = [_tlisi64(*imgs[k:k + 3], t) for k in range(case["snaps"] - 2)]
            if op == "sequence":
                return torch.stack(m)
            return m[0] if op == "pipe_host" else m + imgs
        # A running stream: snapshot k's predecessors are the run's, cyclically.
        c = len(imgs)
        every.append([_tlisi64(imgs[(k - 2) % c], imgs[(k - 1) % c], imgs[k], t)
                      for k in range(c)])
    if op == "batch":
        return [torch.stack(m) for m in every]
    return [m[k] for k in range(case["snaps"]) for m in every]
