"""The calls a user of this package makes, at the sizes they are made at.

Each case is one pass through a public entry point: velocity fields of frame
pairs in device memory (FlctBatch, or the C ABI's flct_gpu_velocity_device as
bench.py calls it), the same from host arrays (flct), one shift of two whole
frames (sigma 0), and the warp program's two computations (warp).

Images and fields are returned as float32: that is what the flct and warp
programs write (the vel_ccor file format of the reference holds float32, and
the kernels' own accuracy is that of FP32).  The mask vm is returned as it is.
exact() is a plain torch restatement in 64 bits of the reference's arithmetic.
"""
import ctypes
import math
import random

import numpy as np
import torch

from pyflct_gb300 import _lib
from pyflct_gb300.flct import FlctBatch, flct, make_params, warp

XMISS = -999999.0
WARP_PI = 3.1415926535898  # the reference warp's pi (warp.c:768)


def _frame(name, call, nx, ny, sigma, skip="", kr=0.0, thresh="", noise=0.0):
    c = {"call": call, "nx": nx, "ny": ny, "sigma": sigma, "skip": skip, "kr": kr, "thresh": thresh, "noise": noise}
    return {"name": name, **c} if name else c


def listed():
    return [
        # a small cut-out, every pixel (the 128 x 128 sigma 4 workload): launches and latency
        _frame("cutout_128", "batch", 128, 128, 4.0),
        # the reference's shipped test: 201 x 101 frames, sigma 5, -k 0.5, from host arrays
        _frame("test_201x101_host", "host", 201, 101, 5.0, kr=0.5),
        # a thresholded and filtered frame, a fifth of its pixels near zero (512^2, -t 0.1a -k 0.5)
        _frame("frame_512_thresh_kr", "batch", 512, 512, 8.0, kr=0.5, thresh="0.1a", noise=0.2),
        # the headline workload: 1024^2, sigma 8, every fourth pixel, interpolated between
        _frame("frame_1024_skip4i", "device", 1024, 1024, 8.0, skip="4i"),
        # the same call from and to host arrays: what a script on numpy frames waits for
        _frame("frame_1024_skip4i_host", "host", 1024, 1024, 8.0, skip="4i"),
        # a ragged frame at sigma 12 (box 48), every pixel
        _frame("frame_769x1023_sigma12", "batch", 769, 1023, 12.0),
        # a campaign of mixed frame pairs in one call (sides 128..768, sigma 3, 5, 8, 12)
        {"name": "campaign_16", "call": "mixed", "pairs": 16, "mix": 4},
        # a large frame at sigma 15 (box 64), every second pixel, interpolated
        _frame("frame_2048_sigma15_skip2i", "batch", 2048, 2048, 15.0, skip="2i"),
        # wide windows: sigma 20 (box 84) on a coarse grid
        _frame("frame_512_sigma20_skip4i", "batch", 512, 512, 20.0, skip="4i"),
        # co-alignment of two whole frames (sigma 0)
        _frame("align_1000x1200", "device", 1000, 1200, 0.0),
        # non-uniform warp of an image along a displacement field
        {"name": "warp_384x512", "call": "warp", "nx": 384, "ny": 512},
        # uniform sub-pixel shift of an image
        {"name": "shift_1000x1536", "call": "shift", "nx": 1000, "ny": 1536},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choices(["batch", "device", "host", "mixed", "align", "warp", "shift"],
                       [40, 18, 16, 8, 4, 7, 7])[0]
    if kind == "mixed":
        return {"call": "mixed", "pairs": _log(rng, 3, 20), "mix": rng.randrange(1 << 20)}
    if kind == "warp":
        return {"call": "warp", "nx": _log(rng, 48, 640), "ny": _log(rng, 48, 640)}
    if kind == "shift":
        return {"call": "shift", "nx": _log(rng, 48, 1600), "ny": _log(rng, 48, 1600)}
    if kind == "align":
        return _frame("", "device", _log(rng, 96, 1200), _log(rng, 96, 1200), 0.0)
    while True:
        big = 2000 if kind != "host" else 1100
        nx, ny = _log(rng, 96, big), _log(rng, 96, big)
        sigma = round(rng.uniform(3.0, 15.9), 1) if rng.random() < 0.9 else round(rng.uniform(16.0, 24.0), 1)
        skip = ""
        n = rng.choice([0, 0, 2, 3, 4, 5, 8])
        if n:
            skip = str(n)
            if rng.random() < 0.3:
                skip += "p%dq%d" % (rng.randrange(n), rng.randrange(n))
            if rng.random() < 0.8:
                skip += "i"
        c = _frame("", kind, nx, ny, sigma, skip=skip, kr=round(rng.uniform(0.3, 0.8), 2) if rng.random() < 0.3 else 0.0)
        if rng.random() < 0.25:
            c["thresh"], c["noise"] = rng.choice(["0.1a", "0.02", "0.05a"]), 0.2
        windows = _windows(nx, ny, skip)
        if windows * _box(nx, ny, sigma) ** 2 <= (2.0e9 if _box(nx, ny, sigma) <= 64 else 1.1e8):
            return c


# ------------------------------------------------------------ geometry ----

def _skip(text):
    """-s N[pP][qQ][i] with P, Q >= 0 -> (N, slow offset, fast offset, interpolate); N = 1: every pixel."""
    if not text:
        return 1, 0, 0, False
    interp = text.endswith("i")
    n, _, pq = text.rstrip("i").partition("p")
    p, _, q = pq.partition("q")
    return int(n), int(q or 0), int(p or 0), interp


def _windows(nx, ny, skip):
    n, xo, yo, _ = _skip(skip)
    return len(range(xo, nx, n)) * len(range(yo, ny, n))


def _half(nx, ny, sigma):
    """Half the sliding box's side (flct.c:567-580)."""
    nt = int(int(sigma) * math.sqrt(math.log(1.0 / 1e-2)))
    return min(nt // 2 * 2, min(nx, ny) // 3 // 2 * 2)


def _box(nx, ny, sigma):
    return 2 * _half(nx, ny, sigma)


def _pairs(case):
    """The frame pairs of a velocity case, each as a case of its own."""
    if case["call"] != "mixed":
        return [case]
    r = random.Random(case["mix"])
    return [_frame("", "batch", r.choice([128, 256, 384, 512, 768]), r.choice([128, 256, 384, 512, 768]),
                   float(r.choice([3, 5, 8, 12]))) for _ in range(case["pairs"])]


# -------------------------------------------------------------- inputs ----

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _field(nx, ny, gen, slope=2.0):
    """Random field with power spectrum ~ k^-slope, unit RMS (synth.kfield on the device)."""
    d = gen.device
    kx = torch.fft.fftfreq(nx, 1.0 / nx, dtype=torch.float64, device=d)[:, None]
    ky = torch.fft.fftfreq(ny, 1.0 / ny, dtype=torch.float64, device=d)[None, :]
    k = torch.sqrt(kx * kx + ky * ky)
    k[0, 0] = 1.0
    amp = k ** (-slope / 2)
    amp[0, 0] = 0.0
    z = torch.randn((nx, ny, 2), dtype=torch.float64, device=d, generator=gen)
    f = torch.fft.ifft2(torch.view_as_complex(z) * amp).real
    return (f / f.square().mean().sqrt()).contiguous()


def _displacement(nx, ny, gen, rms=0.4):
    """Smooth displacement (slow, fast) of the given RMS length."""
    a, b = _field(nx, ny, gen, 4.0), _field(nx, ny, gen, 4.0)
    s = rms / math.sqrt(2.0)
    return a * s, b * s


def _moved(f, ds, df):
    """f(r - d(r)) by periodic cubic convolution."""
    nx, ny = f.shape
    i = torch.arange(nx, dtype=torch.float64, device=f.device)[:, None] - ds
    j = torch.arange(ny, dtype=torch.float64, device=f.device)[None, :] - df
    i0, j0 = torch.floor(i), torch.floor(j)
    out = torch.zeros_like(f)
    for a in range(-1, 3):
        wa = _keys((i - i0 - a).abs())
        ia = (i0.long() + a) % nx
        for b in range(-1, 3):
            out += wa * _keys((j - j0 - b).abs()) * f[ia, (j0.long() + b) % ny]
    return out


def _keys(t):
    return torch.where(t >= 1.0, ((-0.5 * t + 2.5) * t - 4.0) * t + 2.0, (1.5 * t - 2.5) * t * t + 1.0)


def _frames(pair, gen):
    """Two frames of one pair: a red random field and the same field displaced; with `noise` that
    share of the first frame's pixels holds values near zero before the displacement."""
    nx, ny = pair["nx"], pair["ny"]
    f1 = _field(nx, ny, gen)
    if pair.get("noise"):
        low = torch.rand((nx, ny), dtype=torch.float64, device=gen.device, generator=gen)
        val = torch.rand((nx, ny), dtype=torch.float64, device=gen.device, generator=gen) * 0.1 - 0.05
        f1 = torch.where(low < pair["noise"], val, f1)
    if pair["sigma"] <= 0:  # one shift of the whole frame
        d = torch.rand(2, dtype=torch.float64, device=gen.device, generator=gen) * 6.0 - 3.0
        ds, df = d[0].expand(nx, ny), d[1].expand(nx, ny)
    else:
        ds, df = _displacement(nx, ny, gen)
    return f1, _moved(f1, ds, df).contiguous()


def _inputs(case, seed):
    gen = torch.Generator(device=_device())
    gen.manual_seed(int(seed))
    nx, ny = case.get("nx"), case.get("ny")
    if case["call"] == "warp":
        ds, df = _displacement(nx, ny, gen)
        return _field(nx, ny, gen), df, ds
    if case["call"] == "shift":
        d = torch.rand(2, dtype=torch.float64, device=gen.device, generator=gen).tolist()
        return _field(nx, ny, gen), d[0] * 4.0 - 2.0, d[1] * 4.0 - 2.0
    return [_frames(p, gen) for p in _pairs(case)]


def _params(pair):
    return make_params(1.0, 1.0, pair["sigma"], pair["thresh"] or None, pair["kr"] or None, pair["skip"] or None)


def prepare(case, seed):
    call = case["call"]
    x = _inputs(case, seed)
    if call in ("warp", "shift"):
        if call == "warp":
            return {"call": call, "args": [v.cpu().numpy() for v in x]}
        return {"call": call, "args": [x[0].cpu().numpy(), np.array([[x[1]]]), np.array([[x[2]]])]}
    if call == "host":
        kw = {"kr": case["kr"] or None, "thresh": case["thresh"] or None, "skip": case["skip"] or None}
        return {"call": call, "f1": x[0][0].cpu().numpy(), "f2": x[0][1].cpu().numpy(), "sigma": case["sigma"], "kw": kw}
    if call == "device":
        p = _params(case)
        ctx = _lib.context(0)
        n = ctx.lib.flct_gpu_output_len(ctypes.byref(p), case["nx"], case["ny"])
        shape = (case["nx"], case["ny"]) if n == case["nx"] * case["ny"] else (1, 1)
        out = [torch.empty(shape, dtype=torch.float64, device=x[0][0].device) for _ in range(3)]
        return {"call": call, "ctx": ctx, "p": p, "f1": x[0][0], "f2": x[0][1], "nx": case["nx"], "ny": case["ny"], "out": out}
    pairs = _pairs(case)
    b = FlctBatch([(p["nx"], p["ny"]) for p in pairs], [_params(p) for p in pairs])
    for k, (f1, f2) in enumerate(x):
        b.f1[k].copy_(f1)
        b.f2[k].copy_(f2)
    return {"call": call, "batch": b}


def run(state):
    call = state["call"]
    if call in ("warp", "shift"):
        return warp(*state["args"]).astype(np.float32)
    if call == "host":
        vx, vy, vm = flct(state["f1"], state["f2"], 1.0, 1.0, state["sigma"], **state["kw"])
        return [vx.astype(np.float32), vy.astype(np.float32), vm]
    if call == "device":
        ctx, o = state["ctx"], state["out"]
        ctx.check(ctx.lib.flct_gpu_velocity_device(
            ctx.h, ctypes.byref(state["p"]), state["f1"].data_ptr(), state["f2"].data_ptr(), state["nx"], state["ny"],
            o[0].data_ptr(), o[1].data_ptr(), o[2].data_ptr(), torch.cuda.current_stream().cuda_stream))
        return [o[0].float(), o[1].float(), o[2]]
    b = state["batch"]
    b.run()
    return [[vx.float(), vy.float(), vm] for vx, vy, vm in zip(b.vx, b.vy, b.vm)]


def work(case):
    """Frames read and fields written once; the windows' transforms by their operation count
    (three n x n transforms of real images, products, peak); the warp's sum over the half spectrum."""
    if case["call"] in ("warp", "shift"):
        nx, ny = case["nx"], case["ny"]
        n = nx * ny
        if case["call"] == "warp":
            return {"bytes": 32.0 * n, "flops": 4.0 * n * nx * (ny // 2 + 1)}
        return {"bytes": 16.0 * n, "flops": 10.0 * n * math.log2(n)}
    by = fl = 0.0
    for p in _pairs(case):
        n = p["nx"] * p["ny"]
        if p["sigma"] <= 0:
            by, fl = by + 16.0 * n, fl + 7.5 * n * math.log2(n)
            continue
        m = _box(p["nx"], p["ny"], p["sigma"]) ** 2
        w = _windows(p["nx"], p["ny"], p["skip"]) * (1.0 - p["noise"])
        by, fl = by + 40.0 * n, fl + w * (7.5 * m * math.log2(m) + 12.0 * m)
    return {"bytes": by, "flops": fl}


# --------------------------------------------------------------- exact ----

def _wavenumbers(n, device):
    k = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device=device)
    if n % 2 == 0:
        k[n // 2] = n // 2
    return k


def _peak(c):
    """Sub-pixel peak of |c| [m][n0][n1] in the half-shifted frame less the centre (flct.c:1515-1640)."""
    m, n0, n1 = c.shape
    c = torch.roll(c.abs(), (n0 // 2, n1 // 2), (1, 2)).reshape(m, -1)
    at = c.argmax(1)
    i, j = at // n1, at % n1
    inside = (i > 0) & (i < n0 - 1) & (j > 0) & (j < n1 - 1) & (c.gather(1, at[:, None])[:, 0] != 0)
    q = torch.where(inside, at, torch.full_like(at, n1 + 1))
    v = [[c.gather(1, (q + a * n1 + b)[:, None])[:, 0] for b in (-1, 0, 1)] for a in (-1, 0, 1)]
    fx, fy = 0.5 * (v[2][1] - v[0][1]), 0.5 * (v[1][2] - v[1][0])
    fxx, fyy = v[2][1] + v[0][1] - 2 * v[1][1], v[1][2] + v[1][0] - 2 * v[1][1]
    fxy = 0.25 * (v[2][2] + v[0][0] - v[2][0] - v[0][2])
    den = fxy * fxy - fxx * fyy
    zero = torch.zeros_like(fx)
    i = i + torch.where(inside, (fyy * fx - fy * fxy) / den, zero)
    j = j + torch.where(inside, (fxx * fy - fx * fxy) / den, zero)
    empty = c.gather(1, at[:, None])[:, 0] == 0
    return torch.where(empty, zero, i - n0 // 2), torch.where(empty, zero, j - n1 // 2)


def _correlate(a, b, kr):
    n0, n1 = a.shape[-2:]
    c = torch.fft.rfft2(a).conj() * torch.fft.rfft2(b)
    if kr:
        gx = torch.exp(-(_wavenumbers(n0, a.device) / (kr * (n0 // 2))) ** 2)
        gy = torch.exp(-(_wavenumbers(n1, a.device)[: n1 // 2 + 1] / (kr * (n1 // 2))) ** 2)
        c = c * (gx[:, None] * gy[None, :]) ** 2
    return _peak(torch.fft.irfft2(c, (n0, n1)))


def _grid_up(g, nx, ny, n, xo, yo):
    """Cubic convolution of the skip grid at every pixel; XMISS outside it or near a missing value."""
    gx, gy = g.shape
    c = torch.empty((gx + 2, gy + 2), dtype=torch.float64, device=g.device)
    c[1:-1, 1:-1] = g
    c[0, 1:-1], c[-1, 1:-1] = g[2] - 3 * g[1] + 3 * g[0], g[-3] - 3 * g[-2] + 3 * g[-1]
    c[1:-1, 0], c[1:-1, -1] = g[:, 2] - 3 * g[:, 1] + 3 * g[:, 0], g[:, -3] - 3 * g[:, -2] + 3 * g[:, -1]
    c[0, 0], c[-1, 0] = 3 * c[1, 0] - 3 * c[2, 0] + c[3, 0], 3 * c[-2, 0] - 3 * c[-3, 0] + c[-4, 0]
    c[0, -1], c[-1, -1] = 3 * c[0, -2] - 3 * c[0, -3] + c[0, -4], 3 * c[-2, -1] - 3 * c[-3, -1] + c[-4, -1]

    def axis(m, off, count):
        x = (torch.arange(m, dtype=torch.float64, device=g.device) - off) / n
        z = x.clamp(min=0).long().clamp(max=count - 2)
        w = torch.zeros((m, count + 2), dtype=torch.float64, device=g.device)
        s = torch.zeros_like(w)
        for q in range(-1, 3):
            w.scatter_(1, (z + 1 + q)[:, None], _keys((x - (z + q)).abs())[:, None])
            s.scatter_(1, (z + 1 + q)[:, None], 1.0)
        return w, s, (x >= 0) & (x <= count - 1)

    wx, sx, okx = axis(nx, xo, gx)
    wy, sy, oky = axis(ny, yo, gy)
    miss = (c == XMISS).double()
    bad = (sx @ miss @ sy.T > 0) | ~(okx[:, None] & oky[None, :])
    return torch.where(bad, torch.full_like(bad, XMISS, dtype=torch.float64), wx @ c @ wy.T)


def _exact_pair(p, f1, f2):
    nx, ny, dev = p["nx"], p["ny"], f1.device
    if p["sigma"] <= 0:
        a, b = f1 - f1.mean(), f2 - f2.mean()
        si, sj = _correlate(a[None], b[None], p["kr"])
        one = torch.ones((1, 1), dtype=torch.float64, device=dev)
        return [sj.reshape(1, 1), si.reshape(1, 1), one]
    n, xo, yo, interp = _skip(p["skip"])
    t = p["thresh"]
    thr = float(t.rstrip("a")) if t else 0.0
    if t and not t.endswith("a") and 0 < thr < 1:
        thr *= max(float(f1.abs().max()), float(f2.abs().max()))
    grid = torch.zeros((nx, ny), dtype=torch.bool, device=dev)
    grid[xo::n, yo::n] = True
    pix = (grid & (0.5 * (f1 + f2).abs() >= thr)).nonzero()
    half = _half(nx, ny, p["sigma"])
    m = 2 * half
    lo = [torch.minimum((pix[:, k] - (half - 1)).clamp(min=0), torch.full_like(pix[:, k], s - m)) for k, s in ((0, nx), (1, ny))]
    u1, u2 = (f.unfold(0, m, 1).unfold(1, m, 1) for f in (f1, f2))
    ar = torch.arange(m, device=dev)
    vx, vy, vm = (torch.full((nx, ny), XMISS, dtype=torch.float64, device=dev) for _ in range(3))
    step = max(1, (1 << 26) // (m * m))
    for s in range(0, len(pix), step):
        i, j, li, lj = pix[s:s + step, 0], pix[s:s + step, 1], lo[0][s:s + step], lo[1][s:s + step]
        gi = torch.exp(-(((li - i)[:, None] + ar) / p["sigma"]) ** 2)
        gj = torch.exp(-(((lj - j)[:, None] + ar) / p["sigma"]) ** 2)
        g = gi[:, :, None] * gj[:, None, :]
        a, b = u1[li, lj], u2[li, lj]
        si, sj = _correlate((a - a.mean((1, 2), keepdim=True)) * g, (b - b.mean((1, 2), keepdim=True)) * g, p["kr"])
        vx[i, j], vy[i, j] = sj, si
    vm = (vx != XMISS).double()
    if interp:
        for v in (vx, vy):
            v.copy_(torch.where(grid, v, _grid_up(v[xo::n, yo::n], nx, ny, n, xo, yo)))
        vm = torch.where(grid, vm, 0.5 * (vx != XMISS))
    zero = torch.zeros_like(vx)
    return [torch.where(vx == XMISS, zero, vx), torch.where(vy == XMISS, zero, vy), vm]


def _exact_warp(case, x):
    f, df, ds = x
    nx, ny = f.shape
    spec = torch.fft.fft2(f) / (nx * ny)
    kx, ky = _wavenumbers(nx, f.device), _wavenumbers(ny, f.device)
    if case["call"] == "shift":
        px = torch.exp(1j * 2 * WARP_PI * kx * (-ds / nx))
        py = torch.exp(1j * 2 * WARP_PI * ky * (-df / ny))
        return torch.fft.ifft2(spec * px[:, None] * py[None, :], norm="forward").real
    out = torch.empty_like(f)
    j = torch.arange(ny, dtype=torch.float64, device=f.device)
    rows = max(1, (1 << 25) // (ny * max(nx, ny)))
    for i in range(0, nx, rows):
        r = torch.arange(i, min(i + rows, nx), dtype=torch.float64, device=f.device)
        xa = (2 * WARP_PI / nx * (r[:, None] - ds[i:i + rows])).reshape(-1)
        ya = (2 * WARP_PI / ny * (j[None, :] - df[i:i + rows])).reshape(-1)
        ey = torch.polar(torch.ones((), dtype=torch.float64, device=f.device), ya[:, None] * ky)
        ex = torch.polar(torch.ones((), dtype=torch.float64, device=f.device), xa[:, None] * kx)
        out[i:i + rows] = ((ey @ spec.T) * ex).sum(1).real.reshape(-1, ny)
    return out


def exact(case, seed):
    x = _inputs(case, seed)
    if case["call"] in ("warp", "shift"):
        return _exact_warp(case, x).cpu().numpy()
    got = [_exact_pair(p, f1, f2) for p, (f1, f2) in zip(_pairs(case), x)]
    return got if case["call"] in ("batch", "mixed") else got[0]
