"""The calls whose speed matters, as a user's program makes them.

A program that tracks a pair of SLC images keeps one `runtime.Context`, has the
two images in HBM (or in pinned host memory, as read from the files), and calls
`strack`, `strackw`, `strack_batch` or `cull`; results come back as host grids.
Every grid covers the whole image, so its outermost points fall out of bounds
and come back as failures (-2e9), as they do for the command-line tools.

`exact()` restates the same computation in plain torch in 64 bits.
"""
import math

import numpy as np
import torch

from specklesource_b200 import abi, runtime, synth

FAIL = -2.0e9
DEV = "cuda"

_STRACK = dict(kind="strack", host=False, int16=False, amp_only=False, coh_lo=0.6, coh_hi=0.8, dead=0.0)


def listed():
    return [
        # a tile of a mosaic, a quick look: the smallest call in use
        dict(_STRACK, name="strack_256x512_w32", na=256, nr=512, w=32, step_r=16, step_a=8),
        # one burst-sized pair with the default window
        dict(_STRACK, name="strack_1024x2048_w32", na=1024, nr=2048, w=32, step_r=16, step_a=8, dead=0.05),
        # big-endian complex int16 files in pinned host memory, as the tools read them
        dict(_STRACK, name="strack_host_i16_w48", na=2048, nr=4096, w=48, step_r=24, step_a=24, host=True, int16=True,
             dead=0.02),
        # a large scene at full posting, complex window 64
        dict(_STRACK, name="strack_6000x12000_w64", na=6000, nr=12000, w=64, step_r=24, step_a=6, coh_lo=0.3,
             coh_hi=0.9, dead=0.01),
        # detected (amplitude only) tracking, -noComplex
        dict(_STRACK, name="strack_amp_w32", na=1024, nr=2048, w=32, step_r=16, step_a=8, amp_only=True,
             coh_lo=0.8, coh_hi=0.95),
        # half of the scene decorrelated: complex, small and large amplitude tries
        dict(_STRACK, name="strack_fallback_w64", na=2048, nr=4096, w=64, step_r=32, step_a=32, coh_lo=0.2, coh_hi=0.8,
             dead=0.5),
        # fast flow, amplitude search: small, middle and large search windows
        dict(kind="strackw", name="strackw_1024x2048_w64", na=1024, nr=2048, w=64, pad=8, step_r=24, step_a=24, navg=1),
        dict(kind="strackw", name="strackw_2048x4096_w128", na=2048, nr=4096, w=128, pad=32, step_r=48, step_a=48,
             navg=2),
        dict(kind="strackw", name="strackw_2000x4000_w224", na=2000, nr=4000, w=224, pad=48, step_r=32, step_a=32,
             navg=2),
        # many small tiles of mixed windows in one call
        dict(kind="batch", name="batch_24_tiles", tiles=24, lo=512, hi=1024, dead=0.03),
        # culling the grid of a burst-sized pair (tool defaults) and of a large scene
        dict(kind="cull", name="cull_119x124", na=119, nr=124, box=9, n_good=17, sr=2, sa=8, island=-1),
        dict(kind="cull", name="cull_1969x993", na=1969, nr=993, box=5, n_good=12, sr=3, sa=3, island=10),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["strack", "strack", "strack", "strackw", "strackw", "batch", "cull"])
    if kind == "strack":
        w = rng.choice([16, 24, 32, 48, 64])
        na, nr = log(256, 4000), log(512, 8000)
        mode = rng.choice(["plain", "plain", "host", "amp", "fallback"])
        # at most 60,000 points, 6,000 where every point may need the larger windows
        most = 60000 if mode in ("plain", "host") else 6000
        sa = max(rng.randint(w // 8, w), 1)
        sr = max(rng.randint(w // 4, w), na * nr // (sa * most) + 1)
        c = dict(_STRACK, na=na, nr=nr, w=w, step_r=sr, step_a=sa, dead=round(rng.uniform(0.01, 0.05), 3))
        if mode == "host":
            c.update(host=True, int16=rng.random() < 0.5)
        elif mode == "amp":
            c.update(amp_only=True, dead=0.0, coh_lo=0.8, coh_hi=0.95)
        elif mode == "fallback":
            c.update(coh_lo=0.2, coh_hi=0.8, dead=round(rng.uniform(0.2, 0.8), 2))
        return c
    if kind == "strackw":
        w = rng.choice([32, 48, 64, 96, 128, 192, 224, 256])
        na, nr = log(max(512, 3 * w), 2000), log(max(1024, 3 * w), 4000)
        step = max(rng.randint(16, 48), int(math.sqrt(na * nr / 4000)) + 1)
        return dict(kind="strackw", na=na, nr=nr, w=w, pad=rng.randint(5, max(6, w // 2 - 16)), step_r=step, step_a=step,
                    navg=rng.choice([1, 2, 3]))
    if kind == "batch":
        lo = rng.randint(300, 512)
        return dict(kind="batch", tiles=rng.randint(4, 32), lo=lo, hi=lo + rng.randint(64, 512),
                    dead=round(rng.uniform(0.01, 0.05), 3))
    box = rng.choice([5, 7, 9])
    return dict(kind="cull", na=log(60, 1500), nr=log(60, 1000), box=box, n_good=box * box // 5, sr=rng.randint(1, 5),
                sa=rng.randint(1, 8), island=rng.choice([-1, 5, 10]))


# ---------------------------------------------------------------- inputs

BULK_R, BULK_A = 3.0, -2.0  # the offset the orbits predict, given as the initial shift


def _blocks(case, seed):
    """Coherence: its level by 512-pixel blocks, and a `dead` share of 128-pixel blocks (water, melt) decorrelated."""
    g = torch.Generator().manual_seed(seed)
    nb, mb = case["na"] // 128 + 1, case["nr"] // 128 + 1
    level = torch.rand(nb // 4 + 1, mb // 4 + 1, generator=g, dtype=torch.float64)
    coh = case["coh_lo"] + (case["coh_hi"] - case["coh_lo"]) * level
    coh = coh.repeat_interleave(4, 0).repeat_interleave(4, 1)[:nb, :mb].contiguous()
    order = torch.randperm(nb * mb, generator=g)[: round(case["dead"] * nb * mb)]
    coh.view(-1)[order] = 0.0
    coh = coh.to(DEV)
    return lambda y, x: coh[(y // 128).long(), (x // 128).long()]


def _inside(case, looks):
    y = torch.arange(0, case["na"], looks, device=DEV)[:, None] / case["na"]
    x = torch.arange(0, case["nr"], looks, device=DEV)[None, :] / case["nr"]
    return x + y > 0.2


def _params(case, **kw):
    w = case["w"]
    if case.get("dead"):  # an ice mask in 8 x 8 looks leaves out a corner of the scene
        m = _inside(case, 8).to(torch.uint8).cpu().numpy()
        kw["mask"] = dict(r0=0, a0=0, nr=m.shape[1], na=m.shape[0], nrl=8, nal=8, mask=m)
    return abi.TrackParams(rStart=w // 2, aStart=w // 2, deltaR=case["step_r"], deltaA=case["step_a"],
                           nR=(case["nr"] - w) // case["step_r"] + 1, nA=(case["na"] - w) // case["step_a"] + 1,
                           wR=w, wA=w, wRa=w, wAa=w, rShiftPoly=(BULK_R, 0.0, 0.0), aShiftPoly=(BULK_A, 0.0, 0.0),
                           **kw)


def _strack_pair(case, seed):
    s1, s2 = synth.make_pair(case["na"], case["nr"], seed,
                             dr=lambda y, x: BULK_R + 1.5 * torch.sin(2 * math.pi * x / 1500),
                             da=lambda y, x: BULK_A + 0.5 * torch.cos(2 * math.pi * y / 900),
                             coherence=_blocks(case, seed), device=DEV)
    if case["dead"] == 0.0 and not case["amp_only"]:
        # the corner outside the swath holds zeros
        inside = _inside(case, 1)
        s1, s2 = s1 * inside, s2 * inside
    if case["int16"]:
        s1, s2 = [torch.view_as_real(s).mul(300).round().clamp(-32767, 32767).to(torch.int16) for s in (s1, s2)]
    return s1.contiguous(), s2.contiguous()


def _as_file(t):
    """A device image as the bytes of its (big-endian) file in pinned host memory."""
    if t.dtype == torch.complex64:
        t = torch.view_as_real(t)
    item = t.element_size()
    raw = t.contiguous().view(torch.uint8).reshape(-1, item).flip(1).reshape(-1)
    host = torch.empty(raw.shape, dtype=torch.uint8, pin_memory=True)
    host.copy_(raw)
    if item == 2:
        return host.numpy().view(">i2").reshape(t.shape)
    return host.numpy().view(">c8").reshape(t.shape[:2])


def _strackw_pair(case, seed):
    """A shear zone; the flow stays well inside the search radius."""
    most = min(0.6 * case["pad"], 40.0)
    ph = 0.01 * (seed % 628)

    def flow(a, y, x):
        return a * torch.tanh((x - 2 * y) / 1500.0 + torch.sin(x / 700 + ph))

    return synth.make_pair(case["na"], case["nr"], seed, dr=lambda y, x: BULK_R + flow(most, y, x),
                           da=lambda y, x: BULK_A + flow(0.25 * most, y, x), coherence=0.6, device=DEV)


def _tiles(case, seed):
    rng = np.random.default_rng(1000 * case["lo"] + case["hi"] + case["tiles"])  # sizes: the case's own
    out = []
    for k in range(case["tiles"]):
        w = [24, 32, 48, 64][k % 4]
        out.append(dict(_STRACK, na=int(rng.integers(case["lo"], case["hi"])), nr=int(rng.integers(case["lo"], case["hi"])),
                        w=w, step_r=max(8, w // 2), step_a=max(8, w // 2), dead=case["dead"], seed=seed + 7919 * k))
    return out


_CTX = []


def _context():
    """The one context that a program keeps."""
    if not _CTX:
        _CTX.append(runtime.Context(0))
    return _CTX[0]


def prepare(case, seed):
    ctx = _context()
    if case["kind"] == "strack":
        s1, s2 = _strack_pair(case, seed)
        if case["host"]:
            s1, s2 = _as_file(s1), _as_file(s2)
        return dict(kind="strack", ctx=ctx, p=_params(case, noComplex=int(case["amp_only"])), img=(s1, s2))
    if case["kind"] == "strackw":
        p = _params(case, edgePadR=case["pad"], edgePadA=case["pad"], navgR=case["navg"], navgA=case["navg"])
        return dict(kind="strackw", ctx=ctx, p=p, img=_strackw_pair(case, seed))
    if case["kind"] == "batch":
        tiles = _tiles(case, seed)
        pairs = [_strack_pair(t, t["seed"]) for t in tiles]
        return dict(kind="batch", ctx=ctx, p=[_params(t) for t in tiles], img=list(zip(*pairs)))
    grids = synth.offsets_field(case["na"], case["nr"], seed)
    p = abi.CullParams(nR=case["nr"], nA=case["na"], bR=case["box"], bA=case["box"], nGood=case["n_good"],
                       sR=case["sr"], sA=case["sa"], islandThresh=case["island"])
    return dict(kind="cull", ctx=ctx, p=p, grids=grids)


def run(state):
    ctx = state["ctx"]
    if state["kind"] == "strack":
        return ctx.strack(state["p"], *state["img"])
    if state["kind"] == "strackw":
        r = ctx.strackw(state["p"], *state["img"])
        return {k: v for k, v in r.items() if v is not None}
    if state["kind"] == "batch":
        res = ctx.strack_batch(state["p"], *state["img"])
        return {k: np.concatenate([r[k].ravel() for r in res]) for k in ("offR", "offA", "corr", "azd", "type")}
    r = ctx.cull(state["p"], *state["grids"])
    return {k: r[k] for k in ("offR", "offA", "type", "offRS", "offAS", "sigmaR", "sigmaA", "nCulled", "nIslands",
                              "nIslandPoints")}


# ---------------------------------------------------------------- work


def _fft2(n):
    return 10.0 * n * n * math.log2(n)  # 5 N log2 N, N = n^2


def _strack_flops(case):
    w = case["w"]
    peak = _fft2(8) + _fft2(96)
    cmplx = 2 * _fft2(w) + _fft2(2 * w) + peak

    def amp(s):  # two spectra, two detected images, two real transforms, one inverse
        return 2 * _fft2(s) + 4 * _fft2(2 * s) + peak

    if case["amp_only"]:
        return amp(w)
    return cmplx + case["dead"] * (amp(w) + amp(2 * w))


def _points(case):
    return ((case["nr"] - case["w"]) // case["step_r"] + 1) * ((case["na"] - case["w"]) // case["step_a"] + 1)


def work(case):
    if case["kind"] == "cull":
        # offsets, corr, type in; culled and smoothed offsets, sigmas, type out
        n = case["na"] * case["nr"]
        return {"bytes": n * (13.0 + 25.0), "flops": n * (3 * 2.0 * case["box"] ** 2 + 2 * 81 * 12 + 4.0 * case["sr"] * case["sa"])}
    if case["kind"] == "batch":
        both = [work(t) for t in _tiles(case, 0)]
        return {k: sum(b[k] for b in both) for k in ("bytes", "flops")}
    n = _points(case)
    if case["kind"] == "strackw":
        w = case["w"]
        flops = 2 * _fft2(w) + 2 * _fft2(2 * w) + 2 * _fft2(2 * w)
        return {"bytes": 16.0 * case["na"] * case["nr"] + 13.0 * n, "flops": n * flops}
    item = 4 if case["int16"] else 8
    return {"bytes": 2.0 * item * case["na"] * case["nr"] + 17.0 * n, "flops": n * _strack_flops(case)}


# ---------------------------------------------------------------- 64-bit values: tracking


def _windows(img, a, r, w):
    """(n, w, w) complex128 windows at rows a, columns r; zeros outside the image."""
    if img.dtype == torch.int16:
        img = torch.complex(img[..., 0].float(), img[..., 1].float())
    k = torch.arange(w, device=DEV)
    y, x = (a[:, None] + k)[:, :, None], (r[:, None] + k)[:, None, :]
    inside = (y >= 0) & (y < img.shape[0]) & (x >= 0) & (x < img.shape[1])
    v = img[y.clamp(0, img.shape[0] - 1), x.clamp(0, img.shape[1] - 1)]
    return torch.where(inside, v, torch.zeros((), dtype=v.dtype, device=DEV)).to(torch.complex128)


def _doppler(z1, z2):
    """Azimuth carrier of both windows, as a roll of the spectrum in rows."""
    w = z1.shape[1]
    ang = 0.0
    for z in (z1, z2):
        z = z - z.mean((1, 2), keepdim=True)
        ang = ang + torch.angle((z[:, 1:] * z[:, :-1].conj()).sum((1, 2)))
    v = (w // 2) * ang * 0.5 / math.pi
    s = torch.where(v >= 0, (v + 0.5).trunc(), (v - 0.5).trunc()).long()
    return torch.where(s < 0, s + w, s)


def _pad2(f, roll):
    """The spectrum rolled by `roll` rows and zero padded to twice its size (the Nyquist bins go to the negative side)."""
    n, w, _ = f.shape
    rows = (torch.arange(w, device=DEV)[None, :] + roll[:, None]) % w
    f = torch.gather(f, 1, rows[:, :, None].expand(-1, -1, w))
    out = torch.zeros(n, 2 * w, 2 * w, dtype=f.dtype, device=DEV)
    h = w // 2
    for i, i1 in ((slice(0, h), slice(0, h)), (slice(h, w), slice(2 * w - h, 2 * w))):
        for j, j1 in ((slice(0, h), slice(0, h)), (slice(h, w), slice(2 * w - h, 2 * w))):
            out[:, i1, j1] = f[:, i, j]
    return out


def _surface(c):
    """|c| with the zero lag in the middle, and its largest position (rejected near the edge)."""
    m = torch.fft.fftshift(c.abs(), dim=(1, 2))
    n = m.shape[1]
    at = m.reshape(m.shape[0], -1).argmax(1)
    i, j = at // n, at % n
    bad = (i < 4) | (i > n - 4) | (j < 4) | (j > n - 4)
    return m, i, j, bad


def _around(m, i, j, di, dj):
    n = m.shape[1]
    y = (i[:, None] + di).clamp(0, n - 1)[:, :, None]
    x = (j[:, None] + dj).clamp(0, n - 1)[:, None, :]
    return m[torch.arange(m.shape[0], device=DEV)[:, None, None], y, x]


def _oversample(m, i, j):
    """Peak of the 8 x 8 block around (i, j) oversampled 12 times: value, position in 1/12 samples."""
    k = torch.arange(-4, 4, device=DEV)
    f = k.double()
    t, n = torch.arange(8, device=DEV).double(), torch.arange(24, 72, device=DEV).double()
    a = torch.exp(2j * math.pi * (n[:, None] - 12 * t[None, :])[..., None] * f / 96).sum(-1)
    o = (a @ _around(m, i, j, k, k).to(torch.complex128) @ a.T).abs().reshape(len(i), -1)
    v, at = o.max(1)
    return v, 12 * i + at // 48 + 24 - 48, 12 * j + at % 48 + 24 - 48


def _gauss_width(y, x0):
    """Width of a Gaussian fitted to 18 samples: at most five Levenberg-Marquardt steps."""
    y = y / y.max(1, keepdim=True).values
    x = x0[:, None] + torch.arange(18, device=DEV).double()
    n = len(x0)
    a = torch.stack([torch.ones(n, device=DEV, dtype=torch.float64), x[:, 9], torch.full((n,), 2.0, device=DEV, dtype=torch.float64)], 1)

    def model(a):
        t, s = x - a[:, 1:2], a[:, 2:3]
        e = torch.exp(-0.5 * t * t / (s * s))
        v = a[:, 0:1] * e
        d = torch.stack([e, v * t / (s * s), v * t * t / (s * s * s)], 2) * 10
        r = (y - v) * 10
        return d.transpose(1, 2) @ d, (d.transpose(1, 2) @ r[..., None])[..., 0], (r * r).sum(1)

    al, be, chi = model(a)
    lam = torch.full((n,), 0.001, device=DEV, dtype=torch.float64)
    last = torch.full((n,), 2e9, device=DEV, dtype=torch.float64)
    live = torch.ones(n, dtype=torch.bool, device=DEV)
    for _ in range(5):
        cov = al + torch.diag_embed(al.diagonal(dim1=1, dim2=2) * lam[:, None])
        step, info = torch.linalg.solve_ex(cov, be)
        live = live & (info == 0)
        t = a + torch.where(live[:, None], step, 0.0)
        al1, be1, chi1 = model(t)
        up = live & (chi1 < chi)
        a, be, al = torch.where(up[:, None], t, a), torch.where(up[:, None], be1, be), torch.where(up[:, None, None], al1, al)
        chi = torch.where(up, chi1, chi)
        lam = torch.where(up, lam * 0.1, torch.where(live, lam * 10, lam))
        live = live & ~((a[:, 1] - last).abs() < 0.001)
        last = torch.where(live, a[:, 1], last)
    return 0.5 * a[:, 2]


def _widths(m, i, j):
    """Azimuth over range width of the peak through (i, j)."""
    k = torch.arange(-9, 9, device=DEV)
    z = torch.zeros(1, dtype=torch.long, device=DEV)
    rg = _gauss_width(_around(m, i, j, z, k)[:, 0, :], (j - 9).double())
    az = _gauss_width(_around(m, i, j, k, z)[:, :, 0], (i - 9).double())
    return az / rg


def _complex_try(case, img, r1, a1, r2, a2):
    w = case["w"]
    z1, z2 = _windows(img[0], a1, r1, w), _windows(img[1], a2, r2, w)
    if not case["int16"]:
        z1, z2 = z1 * 1000, z2 * 1000
    h = 0.5 * (1 + np.cos(2 * math.pi * np.arange(w // 2) / (w - 1)))
    h = torch.as_tensor(np.concatenate([h[::-1], h]), device=DEV)
    z2 = z2 * (h[:, None] * h[None, :]).float().double()
    p1, p2 = z1.abs().square(), z2.abs().square()
    thr = 1e-9 if case["int16"] else 1e-15
    data = ((p1 < thr) | (p2 < thr)).sum((1, 2)) <= 20
    p1, p2 = p1.mean((1, 2)), p2.mean((1, 2))
    data &= (p1 >= thr) & (p2 >= thr)
    roll = _doppler(z1, z2)
    c = torch.fft.ifft2(_pad2(torch.fft.fft2(z1) * torch.fft.fft2(z2).conj(), roll), norm="forward")
    m, i, j, bad = _surface(c)
    v, io, jo = _oversample(m, i, j)
    cc = torch.where(bad, -1.0, 1.5 * v / 64 / (torch.sqrt(p1 * p2) * float(w) ** 4))
    io, jo = torch.where(bad, -1000, io), torch.where(bad, -1000, jo)
    iq, jq = torch.div(io, 12, rounding_mode="trunc"), torch.div(jo, 12, rounding_mode="trunc")
    gate = (iq >= 9) & (iq + 9 < 2 * w) & (jq >= 9) & (jq + 9 < 2 * w)
    azd = torch.where(gate, _widths(m, iq.clamp(9, 2 * w - 10), jq.clamp(9, 2 * w - 10)), FAIL)
    rs, as_ = (jo.double() - 12 * w) / 24, (io.double() - 12 * w) / 24
    good = data & gate & (cc > 0.185) & (rs.abs() < 0.25 * w) & (as_.abs() < 0.25 * w)
    return dict(data=data, good=good, cc=cc, azd=azd, rs=rs, as_=as_, roll=roll)


def _amp_try(case, img, r1, a1, r2, a2, s, roll):
    """Amplitude try with window s; roll None: estimated from the windows."""
    z1, z2 = _windows(img[0], a1, r1, s), _windows(img[1], a2, r2, s)
    if roll is None:
        roll = _doppler(z1, z2)
    az = roll * s // case["w"]
    a, thr = [], 1e-6 if case["int16"] else 1e-15
    low, data = 0, True
    for z in (z1, z2):
        v = torch.fft.ifft2(_pad2(torch.fft.fft2(z), az), norm="forward").abs().square() / (8.0 * float(s) ** 4)
        low = low | (v < thr)
        data = data & (v.sum((1, 2)) >= 1e-6)
        v = v.sqrt()
        a.append(v - v.mean((1, 2), keepdim=True))
    data = data & (low.sum((1, 2)) <= 20)
    p1, p2 = a[0].square().mean((1, 2)), a[1].square().mean((1, 2))
    m, i, j, bad = _surface(torch.fft.ifft2(torch.fft.fft2(a[0]) * torch.fft.fft2(a[1]).conj(), norm="forward"))
    n = 2 * s
    gate = ~bad & (i > 9) & (i < n - 9) & (j > 9) & (j < n - 9)
    azd = _widths(m, i.clamp(9, n - 10), j.clamp(9, n - 10))
    v, io, jo = _oversample(m, i, j)
    cc = torch.where(bad, -1.0, v / (float(n) ** 4 * 64) / torch.sqrt(p1 * p2))
    rs = (torch.where(bad, -1000, jo).double() - 12 * s) / 24
    as_ = (torch.where(bad, -1000, io).double() - 12 * s) / 24
    good = data & (rs.abs() < 0.3 * s) & (as_.abs() < 0.3 * s) & (cc > (0.07 if s == case["w"] else 0.028))
    return dict(data=data, good=good, cc=cc, azd=azd, gate=gate, rs=rs, as_=as_, roll=roll)


def _exact_strack(case, img):
    p, w, na, nr = _params(case), case["w"], case["na"], case["nr"]
    n = p.nR * p.nA
    k = torch.arange(n, device=DEV)
    cr, ca = p.rStart + (k % p.nR) * p.deltaR, p.aStart + (k // p.nR) * p.deltaA
    br, ba = int(BULK_R), int(BULK_A)
    out = {q: torch.full((n,), v, device=DEV, dtype=torch.float64)
           for q, v in (("offR", FAIL), ("offA", FAIL), ("corr", 0.0), ("azd", 0.0))}

    def within(s):
        r, a = cr - s // 2, ca - s // 2
        ok = (r > 0) & (r + s < nr) & (a > 0) & (a + s < na)
        return ok & (r + br > 0) & (r + br + s < nr) & (a + ba > 0) & (a + ba + s < na)

    def chunks(todo, s):
        q = todo.nonzero()[:, 0]
        return q.split(max(16, int(2.5e7) // (4 * s * s))) if len(q) else ()

    roll = torch.zeros(n, dtype=torch.long, device=DEV)
    todo = torch.ones(n, dtype=torch.bool, device=DEV)
    if case["dead"]:
        todo = _inside(case, 8)[ca // 8, cr // 8]

    def take(q, t):
        out["offR"][q] = torch.where(t["good"], br - t["rs"], out["offR"][q])
        out["offA"][q] = torch.where(t["good"], ba - t["as_"], out["offA"][q])
        todo[q] = t["data"] & ~t["good"]

    if not case["amp_only"]:
        for q in chunks(todo & within(w), w):
            t = _complex_try(case, img, cr[q] - w // 2, ca[q] - w // 2, cr[q] - w // 2 + br, ca[q] - w // 2 + ba)
            out["corr"][q] = torch.where(t["data"], t["cc"], 0.0)
            out["azd"][q] = torch.where(t["data"], t["azd"], 0.0)
            roll[q] = torch.where(t["data"], t["roll"], 0)
            take(q, t)
    for s in (w, 2 * w):
        out["corr"][todo & ~within(s)] = 0.0
        for q in chunks(todo & within(s), s):
            t = _amp_try(case, img, cr[q] - s // 2, ca[q] - s // 2, cr[q] - s // 2 + br, ca[q] - s // 2 + ba, s,
                         None if case["amp_only"] and s == w else roll[q])
            out["corr"][q] = torch.where(t["data"], t["cc"], 0.0)
            out["azd"][q] = torch.where(t["data"] & t["gate"], t["azd"], out["azd"][q])
            roll[q] = t["roll"]
            take(q, t)
    return {q: v.cpu().numpy().reshape(p.nA, p.nR) for q, v in out.items()}


def _exact_strackw(case, img):
    w, na, nr, g = case["w"], case["na"], case["nr"], case["navg"]
    p, n, e, half = _params(case), 2 * w, case["pad"] + 5, 10
    br, ba = int(BULK_R), int(BULK_A)
    k = torch.arange(p.nR * p.nA, device=DEV)
    cr, ca = (k % p.nR) * p.deltaR, (k // p.nR) * p.deltaA
    out = {q: torch.full((len(k),), v, device=DEV, dtype=torch.float64) for q, v in (("offR", FAIL), ("offA", FAIL), ("corr", 0.0))}
    ok = (cr > 0) & (cr < nr) & (ca > 0) & (ca < na) & (cr + br > 0) & (cr + br < nr) & (ca + ba > 0) & (ca + ba < na)
    c2, lags = n - 4 * e, 4 * e + 1  # chip and lags in the doubled image
    box = torch.arange(-g, g + 1, device=DEV)

    def smooth(v, first, size, last):
        if g <= 1:
            return v[:, first:first + size, first:first + size]
        at = (torch.arange(first, first + size, device=DEV)[:, None] + box).clamp(0, last)
        v = sum(v[:, :, at[:, b]] for b in range(2 * g + 1))
        return sum(v[:, at[:, b], :] for b in range(2 * g + 1))

    nn, t = torch.arange(-32, 32, device=DEV).double() + 168, torch.arange(21, device=DEV).double()
    f = torch.arange(1, 11, device=DEV).double()
    ker = 1 + 2 * torch.cos(2 * math.pi * (nn[:, None] - 16 * t[None, :])[..., None] * f / 336).sum(-1)
    for q in ok.nonzero()[:, 0].split(max(4, int(4e6) // (n * n))):
        z1, z2 = _windows(img[0], ca[q], cr[q], w), _windows(img[1], ca[q] + ba, cr[q] + br, w)
        roll = _doppler(z1, z2)
        v1, v2 = [torch.fft.ifft2(_pad2(torch.fft.fft2(z), roll), norm="forward").abs().square() / float(w) ** 4 for z in (z1, z2)]
        big = smooth(v1, 0, n, n - 1).sqrt()
        chip = smooth(v2, 2 * e, c2, 2 * e + c2 + g - 1).sqrt()
        m2 = c2 * c2
        sig = chip.square().sum((1, 2)) / (m2 - 1) - chip.mean((1, 2)).square()
        emb = torch.zeros_like(big)
        emb[:, :c2, :c2] = chip - chip.mean((1, 2), keepdim=True)
        cov = torch.fft.irfft2(torch.fft.rfft2(big) * torch.fft.rfft2(emb).conj(), s=(n, n))[:, :lags, :lags] / m2

        def sums(v):
            s = torch.nn.functional.pad(v.cumsum(1).cumsum(2), (1, 0, 1, 0))
            return (s[:, c2:, c2:] - s[:, :-c2, c2:] - s[:, c2:, :-c2] + s[:, :-c2, :-c2])

        var = sums(big.square()) / (m2 - 1) - (sums(big) / m2).square()
        ncc = cov / (sig[:, None, None] * var).sqrt()
        inner = ncc[:, half:lags - half, half:lags - half]
        v, at = inner.reshape(len(q), -1).max(1)
        i, j = at // inner.shape[2] + half, at % inner.shape[2] + half
        d = torch.arange(-10, 11, device=DEV)
        b = ncc[torch.arange(len(q), device=DEV)[:, None, None], (i[:, None] + d)[:, :, None], (j[:, None] + d)[:, None, :]]
        o = (ker @ b @ ker.T).square().reshape(len(q), -1)
        top, at = o.max(1)
        io, jo = 16 * i + at // 64 + 136 - 160, 16 * j + at % 64 + 136 - 160
        good = v >= 0
        out["corr"][q] = torch.where(good, top.sqrt() / 441, 0.0)
        out["offR"][q] = torch.where(good, br - (jo.double() - 32 * e) / 32, FAIL)
        out["offA"][q] = torch.where(good, ba - (io.double() - 32 * e) / 32, FAIL)
    return {q: v.cpu().numpy().reshape(p.nA, p.nR) for q, v in out.items()}


# ---------------------------------------------------------------- 64-bit values: culling


def _boxes(v, k, nr, ha, hr, fill):
    """Values of the (2 ha + 1) x (2 hr + 1) boxes around the points k; `fill` outside the grid."""
    v = torch.nn.functional.pad(v, (hr, hr, ha, ha), value=fill)
    i, j = k // nr, k % nr
    di, dj = torch.arange(2 * ha + 1, device=DEV), torch.arange(2 * hr + 1, device=DEV)
    return v[(i[:, None] + di)[:, :, None], (j[:, None] + dj)[:, None, :]].reshape(len(k), -1)


def _median_pass(case, R, A):
    """One in-place raster-order median pass, as the fixed point of its decisions."""
    na, nr, h = case["na"], case["nr"], case["box"] // 2
    n = na * nr
    lim = float(np.float32(1 - 2000000000))
    valid = (R > lim) & (A > lim)
    out = torch.zeros(na, nr, dtype=torch.bool, device=DEV)
    before = torch.arange((2 * h + 1) ** 2, device=DEV) < (2 * h + 1) * h + h
    todo = torch.arange(n, device=DEV)
    while len(todo):
        flips = []
        for k in todo.split(1 << 17):
            ok = _boxes(valid, k, nr, h, h, False) & ~(before & _boxes(out, k, nr, h, h, False))
            cnt = ok.sum(1)
            at = (cnt // 2 - 1).clamp(min=0)[:, None]
            far = torch.zeros(len(k), dtype=torch.bool, device=DEV)
            for v, most in ((R, 0.75), (A, 1.0)):
                srt = torch.where(ok, _boxes(v, k, nr, h, h, 0.0), math.inf).sort(1).values
                far |= (v.reshape(-1)[k] - srt.gather(1, at)[:, 0]).abs() > most
            cull = far | (cnt <= case["n_good"])
            flips.append(k[cull != out.view(-1)[k]])
        flips = torch.cat(flips)
        out.view(-1)[flips] ^= True
        near = torch.zeros(1, 1, na, nr, device=DEV)
        near.view(-1)[flips] = 1.0
        near = torch.nn.functional.max_pool2d(near, 2 * h + 1, 1, h)
        todo = near.view(-1).nonzero()[:, 0]
    return torch.where(out, FAIL, R), torch.where(out, FAIL, A)


def _exact_cull(case, grids):
    na, nr = case["na"], case["nr"]
    R, A = (torch.as_tensor(g, device=DEV).double() for g in grids[:2])
    mt = torch.as_tensor(grids[3], device=DEV).long()
    for _ in range(3):
        R, A = _median_pass(case, R, A)
    lim = float(np.float32(1 - 2000000000))
    valid = (R > lim) & (A > lim)
    sig, sm = [torch.full((na * nr,), FAIL, device=DEV, dtype=torch.float64) for _ in range(2)], []
    ii, jj = (g.double() for g in torch.meshgrid(torch.arange(na, device=DEV), torch.arange(nr, device=DEV), indexing="ij"))
    for k in valid.view(-1).nonzero()[:, 0].split(1 << 13):
        ok = _boxes(valid, k, nr, 4, 4, False).double()
        cnt = ok.sum(1)
        x, y = _boxes(ii, k, nr, 4, 4, 0.0) * ok, _boxes(jj, k, nr, 4, 4, 0.0) * ok
        for v, s in ((R, sig[0]), (A, sig[1])):
            v = torch.where(ok > 0, _boxes(v, k, nr, 4, 4, 0.0), 0.0)
            mean = v.sum(1) / cnt
            base = torch.stack([mean.float().double()[:, None] * ok, x, y], 2)
            # least squares without the directions below 1e-5 of the largest
            e, q = torch.linalg.eigh(base.transpose(1, 2) @ base)
            s2 = e.clamp(min=0).sqrt()
            keep = (s2 >= 1e-5 * s2[:, 2:]) & (s2 > 0)
            proj = (q.transpose(1, 2) @ (base.transpose(1, 2) @ v[..., None]))[..., 0]
            coef = (q @ torch.where(keep, proj / e, 0.0)[..., None])[..., 0]
            fit = (coef[:, :1] * mean[:, None] * ok) + coef[:, 1:2] * x + coef[:, 2:] * y
            res = (v - fit) * ok
            var = res.square().sum(1) / (cnt - 3) - res.sum(1).square() / ((cnt - 3) * cnt)
            s[k] = torch.where(cnt > 8, var.clamp(min=1e-5).sqrt(), FAIL)
    sig = [s.view(na, nr) for s in sig]

    def weights(s):
        m = torch.arange(-(s // 2), s // 2 + 1, device=DEV).double()
        return 1.0 - 0.5 * (m.abs() > s / 2.0 - 0.01).double()

    wa, wr = weights(case["sa"]), weights(case["sr"])
    ker = (wa[:, None] * wr[None, :])[None, None]
    pad = (case["sa"] // 2, case["sr"] // 2)

    def conv(v):
        return torch.nn.functional.conv2d(v[None, None], ker, padding=pad)[0, 0]

    good = conv(valid.double())
    looks = torch.tensor([0.0, 1.0, 0.25, 0.015], device=DEV, dtype=torch.float64)
    looks = conv(valid * looks[mt & 3]).clamp(min=1.0)
    ok = ((good > 1) | (case["sa"] == 1) | (case["sr"] == 1)) & (R > lim) & (sig[1] > lim)
    for v in (R, A):
        sm.append(torch.where(ok, conv(torch.where(valid, v, 0.0)) / good, FAIL))
    sig = [torch.where(ok, s / looks.sqrt(), s) for s in sig]
    if case["island"] > 0:
        lab = torch.where(sm[0] > -1.9e9, torch.arange(1.0, na * nr + 1, device=DEV, dtype=torch.float64).view(na, nr), 0.0)
        lab = torch.where(lab > 0, na * nr + 1 - lab, 0.0)  # components take their first pixel's (largest) number
        while True:
            new = torch.where(lab > 0, torch.nn.functional.max_pool2d(lab[None, None], 3, 1, 1)[0, 0], 0.0)
            if torch.equal(new, lab):
                break
            lab = new
        ids, at = lab.view(-1).unique(return_inverse=True)
        isl = torch.zeros(len(ids), dtype=torch.bool, device=DEV)
        for c in (ii, jj):
            lo = torch.full((len(ids),), 1e9, device=DEV, dtype=torch.float64).scatter_reduce(0, at, c.reshape(-1), "amin")
            hi = torch.full((len(ids),), -1e9, device=DEV, dtype=torch.float64).scatter_reduce(0, at, c.reshape(-1), "amax")
            isl |= (hi - lo) > case["island"]
        small = ~isl
        small[ids == 0] = False
        small[(ids > 0).nonzero()[:1, 0]] = False  # the last component is left as it is
        gone = small[at].view(na, nr)
        sm = [torch.where(gone, FAIL, v) for v in sm]
    names = ("offR", "offA", "offRS", "offAS", "sigmaR", "sigmaA")
    out = {q: v.cpu().numpy() for q, v in zip(names, (R, A, *sm, *sig))}
    return dict(out, type=None, nCulled=None, nIslands=None, nIslandPoints=None)


def exact(case, seed):
    if case["kind"] == "cull":
        return _exact_cull(case, synth.offsets_field(case["na"], case["nr"], seed))
    if case["kind"] == "strackw":
        return dict(_exact_strackw(case, _strackw_pair(case, seed)), type=None, stats=None)
    if case["kind"] == "batch":
        res = [_exact_strack(t, _strack_pair(t, t["seed"])) for t in _tiles(case, seed)]
        return dict({k: np.concatenate([r[k].ravel() for r in res]) for k in ("offR", "offA", "corr", "azd")}, type=None)
    return dict(_exact_strack(case, _strack_pair(case, seed)), type=None, stats=None)
