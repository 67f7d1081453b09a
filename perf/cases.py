"""Performance cases of the eSRRF engine: what its users run, over the sizes they run it at.

A case is a dict of plain values; ``prepare`` makes its inputs and handle, ``run`` is one pass
through the public entry points, ``exact`` the same outputs evaluated in float64 with torch,
``work`` the bytes and operations a pass cannot do without.  Kinds of case:

* ``fht``: one super-resolution block of the 2-D Fourier-interpolated path (an engine handle);
  ``push`` frames per call (0: the whole block), ``host``: numpy frames in and out through
  ``LiveSRRF_CL`` as the plugin calls it, else frames and results in device memory; ``vibration``:
  one shift per frame.
* ``bic``: one block of the 2-D bicubic path with macro-pixel correction.
* ``mfm``: one block of the 3-D multi-focus path (nine planes on one camera frame).
* ``sweep``: a batched parameter sweep over uneven blocks.
* ``adjoint``: the re-blur fidelity loss with all its gradients (parameter search).
* ``shifts``: drift estimation of a block against its first frame.
"""
from __future__ import annotations

import ctypes
import math
import pathlib
import sys

import numpy as np
import torch

sys.path.insert(0, str(pathlib.Path(__file__).resolve().parent.parent / "nanoj-esrrf_b200"))
import esrrf  # noqa: E402
from esrrf import lib  # noqa: E402

DEV = "cuda:0"


def _fht(name, w, h, frames, mag, radius, sens, u16=True, weighting=True, push=0, host=False, vibration=False):
    return {"name": name, "kind": "fht", "width": w, "height": h, "frames": frames, "mag": mag, "radius": radius,
            "sens": sens, "u16": u16, "weighting": weighting, "push": push, "host": host, "vibration": vibration}


def listed():
    return [
        # The preview of a live acquisition: a small region, host frames in, host images out.
        _fht("preview_64_m5", 64, 64, 100, 5, 1.5, 1, host=True),
        # Frames handed over one at a time as the camera delivers them, a short rolling block.
        _fht("stream_128_m4", 128, 128, 10, 4, 1.5, 2, push=1),
        # The standard analysis: one rolling block of a 512 x 512 camera region.
        _fht("block_512_m4", 512, 512, 100, 4, 1.5, 2),
        # The plugin's default settings (M 5, radius 2, sensitivity 1) on a ragged float crop.
        _fht("default_299x203_m5", 299, 203, 100, 5, 2.0, 1, u16=False),
        # A large field at full magnification: 4096 x 4096 output.
        _fht("field_1024_m4", 1024, 1024, 40, 4, 1.5, 2),
        # A wide non-square field, low magnification, wide radius, no intensity weighting.
        _fht("wide_640x360_m2_r3", 640, 360, 200, 2, 3.0, 1, weighting=False),
        # Vibration correction on: every frame has its own shift.
        _fht("vibration_256_m4", 256, 256, 100, 4, 1.5, 2, vibration=True),
        # The analysis with "Fourier interpolation" off.
        {"name": "bicubic_512_m4", "kind": "bic", "width": 512, "height": 512, "frames": 100, "mag": 4,
         "radius": 1.5, "sens": 2, "u16": True},
        # A multi-focus microscope: nine planes, 40 timepoints.
        {"name": "mfm_9x128_m3", "kind": "mfm", "width": 128, "height": 128, "frames": 40, "mag": 3, "radius": 1.5,
         "sens": 1, "u16": True},
        # The parameter sweep that users run before an analysis.
        {"name": "sweep_256", "kind": "sweep", "width": 256, "height": 256, "frames": 100, "mags": "2,4",
         "radii": "1.0,1.5,2.5", "senses": "1,2,3", "u16": True},
        # One step of the gradient search that replaces the sweep.
        {"name": "adjoint_128_m4", "kind": "adjoint", "width": 128, "height": 128, "frames": 60, "mag": 4,
         "radius": 1.5, "sens": 2.0, "sigma": 1.5},
        # The shifts that vibration correction uses, estimated from the block itself.
        {"name": "shifts_512", "kind": "shifts", "width": 512, "height": 512, "frames": 100, "u16": True},
    ]


MOST_WORK = 1.5e11  # taps x output pixels x frames of a drawn case (field_1024_m4: 1.7e11)


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["fht"] * 6 + ["bic", "mfm", "sweep", "adjoint", "shifts"])
    w = log_int(48, 900)
    c = {"kind": kind, "width": w, "height": max(40, int(w * rng.uniform(0.5, 1.0))), "frames": log_int(10, 200),
         "mag": rng.choice([2, 3, 4, 5]), "radius": rng.choice([0.5, 1.0, 1.25, 1.5, 2.0, 2.5, 3.0]),
         "sens": rng.choice([1, 1, 2, 3, 4]), "u16": rng.random() < 0.7}
    if kind == "fht":
        c.update(weighting=rng.random() < 0.8, push=rng.choice([0, 0, 0, 1, 7]), host=False,
                 vibration=rng.random() < 0.2)
    elif kind == "mfm":
        c.update(width=log_int(24, 160), height=log_int(24, 160), mag=rng.choice([2, 3, 4]),
                 frames=log_int(8, 60), radius=rng.choice([1.0, 1.5, 2.0]))
    elif kind == "sweep":
        r0 = rng.choice([0.5, 1.0, 1.5])
        c.update(width=log_int(48, 256), height=log_int(48, 256), frames=log_int(20, 150),
                 mags=rng.choice(["2", "3", "4", "2,4", "2,3"]), radii="%g,%g" % (r0, r0 + 1.0),
                 senses=rng.choice(["1", "1,2", "1,2,4"]))
        del c["mag"], c["radius"], c["sens"]
    elif kind == "adjoint":
        c.update(width=log_int(32, 200), height=log_int(32, 200), frames=log_int(10, 80), mag=rng.choice([2, 3, 4]),
                 radius=rng.choice([1.0, 1.3, 1.5, 1.8]), sens=rng.choice([1.0, 1.5, 2.0]),
                 sigma=rng.choice([1.0, 1.5, 2.5]))
        del c["u16"]
    elif kind == "shifts":
        for k in ("mag", "radius", "sens"):
            del c[k]
    while _taps_done(c) > MOST_WORK:
        if c["frames"] > 12:
            c["frames"] = max(10, int(c["frames"] * 0.7))
        else:
            c["width"], c["height"] = max(40, int(c["width"] * 0.8)), max(40, int(c["height"] * 0.8))
    return c


# --------------------------------------------------------------------------------- inputs


def _stack(seed, frames, h, w, planes=1):
    """Blinking emitters along filaments, pixel-sampled Gaussian spots, Poisson and read noise:
    [frames][h][w] (planes > 1: [frames][planes][h][w]) float32 whole numbers on the GPU."""
    g = torch.Generator(device=DEV).manual_seed(int(seed))

    def rand(*s):
        return torch.rand(*s, generator=g, device=DEV)

    n = max(24, int(0.02 * w * h))
    fil = torch.randint(0, 40, (n,), generator=g, device=DEV)
    a, b, t = rand(40, 3), rand(40, 3), rand(n, 1)
    p = a[fil] * (1 - t) + b[fil] * t
    x = p[:, 0] * w + 0.5 * torch.randn(n, generator=g, device=DEV)
    y = p[:, 1] * h + 0.5 * torch.randn(n, generator=g, device=DEV)
    on = torch.empty(frames, n, device=DEV)
    state = (rand(n) < 0.05 / 0.35).float()
    for f in range(frames):
        on[f] = state
        u = rand(n)
        state = torch.where(state > 0, (u >= 0.3).float(), (u < 0.05).float())

    def profile(c, m):
        d = torch.arange(m, device=DEV)[:, None] + 0.5 - c[None]
        return torch.exp(d * d / (-2 * 1.3 ** 2))

    px, py = profile(x, w), profile(y, h)
    out = torch.empty(frames, planes, h, w, device=DEV)
    for z in range(planes):
        pz = torch.exp((z + 0.5 - p[:, 2] * planes) ** 2 / -2.0) if planes > 1 else torch.ones(n, device=DEV)
        for f in range(frames):
            k = on[f] > 0
            out[f, z] = (py[:, k] * (47.0 * pz[k])) @ px[:, k].T
    out = torch.poisson(out + 100.0, generator=g) + 2.0 * torch.randn(out.shape, generator=g, device=DEV) + 100.0
    out = out.round_().clamp_(0, 30000)
    return out[:, 0] if planes == 1 else out


def _shifts(seed, frames):
    """A smooth vibration of up to about a pixel, one (x, y) shift per frame."""
    g = np.random.default_rng(seed)
    t = np.arange(frames)
    sx = 0.9 * np.sin(t * 0.37 + g.uniform(0, 6)) + 0.1 * g.standard_normal(frames)
    sy = 0.7 * np.sin(t * 0.23 + g.uniform(0, 6)) + 0.1 * g.standard_normal(frames)
    return sx.astype(np.float32), sy.astype(np.float32)


ROI = [4, 0, 1, 2, 3, 5, 6, 7, 8]


def _calibration():
    return {"X-shift (pixels)": np.linspace(-0.23, 0.21, 9).astype(np.float32),
            "Y-shift (pixels)": np.linspace(0.13, -0.11, 9).astype(np.float32),
            "Theta (degrees)": np.linspace(-0.53, 0.51, 9).astype(np.float32), "Axial positions": np.zeros(9),
            "ROI #": np.asarray(ROI, np.float32), "Intensity scaling": np.linspace(0.9, 1.1, 9).astype(np.float32),
            "Background level (ADC)": np.full(9, 90.0)}


def _frames(case, seed):
    """The case's frames as float32 whole numbers on the GPU."""
    if case["kind"] != "mfm":
        f = _stack(seed, case["frames"], case["height"], case["width"])
        if case["kind"] == "shifts":
            sx, sy = np.rint(4 * np.stack(_shifts(seed, case["frames"]))).astype(int)
            for t in range(1, case["frames"]):
                f[t] += torch.roll(f[0], (int(sy[t]), int(sx[t])), (0, 1)) // 2
        return f
    p = _stack(seed, case["frames"], case["height"], case["width"], 9)
    n, _, h, w = p.shape
    cam = torch.zeros(n, 3 * h, 3 * w, device=DEV)
    for z, r in enumerate(ROI):
        cam[:, (r // 3) * h:(r // 3 + 1) * h, (r % 3) * w:(r % 3 + 1) * w] = p[:, z]
    return cam


def _list(text, kind):
    return [kind(v) for v in text.split(",")]


def _blocks(frames):
    """Uneven and overlapping rolling blocks."""
    a = max(1, frames * 37 // 100)
    return [(0, a), (a, frames - a), (0, frames)]


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    f = _frames(case, seed)
    n, H, W = f.shape
    s.u16 = bool(case.get("u16"))
    s.frames = f.to(torch.int16) if s.u16 else f
    kind = case["kind"]
    if kind in ("fht", "bic", "mfm"):
        s.eng = esrrf.LiveSRRF_CL()
        s.eng.initialise(W, H, case["mag"], case["radius"], case["sens"], n, n, intWeighting=case.get("weighting", True),
                         doMPmapCorrection=kind != "fht", doFHTinterpolation=kind == "fht", chosenDevice=0,
                         calibTable3DSRRF=_calibration() if kind == "mfm" else None)
        if case.get("host"):
            a = s.frames.cpu().numpy()
            s.host = a.view(np.uint16) if s.u16 else a
        wm, hm, pm = s.eng._shape
        s.out = torch.empty(4, pm, hm, wm, device=DEV)
        s.shift = _shifts(seed, n) if case.get("vibration") else None
    elif kind == "sweep":
        s.sweep = esrrf.Sweep(W, H, n, _list(case["mags"], int), _list(case["radii"], float),
                              _list(case["senses"], int), _blocks(n), device=0)
        s.out = torch.empty(s.sweep.total, device=DEV)
    elif kind == "adjoint":
        s.adj = esrrf.Adjoint(W, H, n, case["mag"], device=0)
    torch.cuda.synchronize()  # the engine's own streams do not wait for torch's
    return s


SLICES = ("AVG", "VAR", "TAC2", "INT")


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def run(s):
    case, kind = s.case, s.case["kind"]
    if kind in ("fht", "bic", "mfm"):
        s.eng.resetFramePosition()
        if s.shift is not None:
            s.eng.loadDriftXYGPUbuffer(*s.shift)
        n = case["frames"]
        step = case.get("push") or n
        if case.get("host"):
            for t in range(0, n, step):
                s.eng.calculateSRRF(s.host[t:t + step])
            o = s.eng.readSRRFbuffer()
            o = o.reshape(4, -1, *o.shape[1:])
        else:
            h = s.eng.handle
            push = lib().esrrf_calculate_srrf_u16_device if s.u16 else lib().esrrf_calculate_srrf_f32_device
            for t in range(0, n, step):
                esrrf._lib.check(h, push(h, _ptr(s.frames[t:]), min(step, n - t)))
            esrrf._lib.check(h, lib().esrrf_read_srrf_device(h, _ptr(s.out)))
            o = s.out
        return {k: o[i] for i, k in enumerate(SLICES)}
    if kind == "sweep":
        h = s.sweep.handle
        esrrf._lib.check(h, lib().esrrf_sweep_run_device(h, _ptr(s.frames), int(s.u16), _ptr(s.out)), sweep=True)
        return _sweep_outputs(case, s.out)
    if kind == "adjoint":
        loss, g, gf = s.adj.loss_and_grad(s.frames, case["radius"], case["sens"], case["sigma"])
        return {"loss": loss, "fwhm": g["fwhm"], "S": g["S"], "sigma": g["sigma"], "frames": gf}
    sx, sy = esrrf.estimate_drift(s.frames)
    return {"x": sx, "y": sy}


def _sweep_outputs(case, flat):
    out, o = {}, 0
    nS, nB = len(_list(case["senses"], int)), len(_blocks(case["frames"]))
    for M in _list(case["mags"], int):
        P = case["height"] * M * case["width"] * M
        for r in _list(case["radii"], float):
            b = flat[o:o + nS * nB * 4 * P].view(nS, nB, 4, case["height"] * M, case["width"] * M)
            o += b.numel()
            for i, k in enumerate(SLICES):
                out["M%d r%g %s" % (M, r, k)] = b[:, :, i]
    return out


# --------------------------------------------------------------------------------- work


def _fht_geometry(M, fwhm):
    """Loop box, squared-distance scale and cut-off of the Fourier path, in the float32 steps that
    define the tap set."""
    f = np.float32
    sigma = f(fwhm) / f(2.354)
    tSS = f(f(f(f(2) * sigma) * f(M)) * sigma) * f(M)
    tSO = f((f(2) * sigma + f(1)) * f(M))
    R = int(f(M) * (f(int(f(2) * sigma)) + f(1)))
    return R, float(tSS), float(tSO)


def _fht_taps(M, fwhm):
    R, _, tSO = _fht_geometry(M, fwhm)
    return [(i, j) for j in range(-R, R + 2) for i in range(-R, R + 2) if 0 < math.hypot(i, j) <= tSO]


def _bic_geometry(fwhm):
    f = np.float32
    sigma = f(fwhm) / f(2.354)
    radius = f(int(f(4) * sigma)) / f(2) + f(1)
    return float(radius), float(f(2) * sigma * sigma), float(f(2) * sigma + f(1))


def _bic_taps(M, fwhm, px, py):
    """(node offset from 2 x cell, displacement) in x and y of a phase's taps on the 2x grid."""
    radius, _, tSO = _bic_geometry(fwhm)
    r0, r1 = -int(2 * radius), int(2 * radius + 1)
    xc, yc = (px + 0.5) / M, (py + 0.5) / M
    kx, ky = int(2 * xc + 1e-9), int(2 * yc + 1e-9)
    got = []
    for j in range(r0, r1 + 1):
        for i in range(r0, r1 + 1):
            dx, dy = (kx + i) / 2 - xc, (ky + j) / 2 - yc
            if dx * dx + dy * dy <= tSO * tSO:
                got.append((kx + i, ky + j, dx, dy))
    return got


def _pixel_taps(case):
    """Taps x output pixels of one frame."""
    kind, px = case["kind"], case["width"] * case["height"]
    if kind == "shifts":
        return px * 63 * 63 / 6
    if kind == "sweep":
        return sum(len(_fht_taps(M, r)) * px * M * M for M in _list(case["mags"], int)
                   for r in _list(case["radii"], float))
    M = case["mag"]
    if kind == "bic":
        return px * sum(len(_bic_taps(M, case["radius"], a, b)) for a in range(M) for b in range(M))
    if kind == "mfm":
        radius, _, tSO = _bic_geometry(case["radius"])
        return 9 * px * M ** 3 * 4 / 3 * math.pi * tSO ** 3 * 4
    return len(_fht_taps(M, case["radius"])) * px * M * M


def _taps_done(case):
    return _pixel_taps(case) * case["frames"] * (4 if case["kind"] == "adjoint" else 1)


def work(case):
    """Frames in and images out once; six operations per tap (a cross product, its weighted
    difference, the inward test, the sum), two multiply-adds per lag for the shifts, and for the
    adjoint one more tap pass."""
    n, px, kind = case["frames"], case["width"] * case["height"], case["kind"]
    flops = _pixel_taps(case) * n * 6
    if kind == "shifts":
        return {"bytes": 2 * n * px, "flops": 2.0 * n * px * 63 * 63}
    if kind == "adjoint":
        return {"bytes": 8 * n * px, "flops": 2.0 * flops}
    per = 2 if case["u16"] else 4
    if kind == "sweep":
        outs = sum(M * M for M in _list(case["mags"], int)) * len(_list(case["radii"], float)) * \
            len(_list(case["senses"], int)) * 3
        return {"bytes": per * n * px + 16 * px * outs, "flops": flops}
    M = case["mag"]
    if kind == "mfm":
        return {"bytes": 9 * px * (per * n + 16 * M ** 3), "flops": flops}
    return {"bytes": px * (per * n + 16 * M * M), "flops": flops}


# --------------------------------------------------------------------------------- float64


def _mirror(n, N):
    """Source index of each sample of a length-n axis mirrored out to N around its centre."""
    tiles = -(-N // n)
    tiles += 1 - tiles % 2
    pos = torch.arange(N) + (tiles * n - N) // 2
    tile, i = pos // n, pos % n
    odd = (tile - (tiles - 1) // 2) % 2 != 0
    return torch.where(odd, n - 1 - i, i)


def _interpolate(raw, M):
    """Fourier (Hartley) interpolation of [f][h][w] float64 frames to [f][h M][w M]."""
    n, h, w = raw.shape
    N = max(1 << (w - 1).bit_length(), 1 << (h - 1).bit_length())
    x = raw[:, _mirror(h, N).to(raw.device)][:, :, _mirror(w, N).to(raw.device)]
    F = torch.fft.fft2(x)
    k = torch.arange(N, device=raw.device)
    k = torch.where(k < N // 2, k, k + (M - 1) * N)
    big = torch.zeros(n, N * M, N * M, dtype=raw.dtype, device=raw.device)
    big = big.index_put((torch.arange(n, device=raw.device)[:, None, None], k[None, :, None], k[None, None, :]),
                        F.real - F.imag)
    G = torch.fft.fft2(big)
    oy, ox = (N * M - h * M) // 2, (N * M - w * M) // 2
    return ((G.real - G.imag) / (N * N))[:, oy:oy + h * M, ox:ox + w * M]


def _before(n, dev):
    return torch.clamp(torch.arange(-1, n - 1, device=dev), min=0)


def _after(n, dev):
    return torch.clamp(torch.arange(1, n + 1, device=dev), max=n - 1)


def _unit_field(I):
    """Unit gradient at every tap source: Roberts cross, x component read one column to the right,
    y component one row down; zero where the gradient is zero."""
    f, H, W = I.shape
    up, left = I[:, _before(H, I.device)], I[:, :, _before(W, I.device)]
    diag = up[:, :, _before(W, I.device)]
    gx = (up - left + I - diag)[:, :, _after(W, I.device)]
    gy = (-up + left + I - diag)[:, _after(H, I.device)]
    m = torch.sqrt(gx * gx + gy * gy)
    safe = torch.where(m > 0, m, torch.ones_like(m))
    return gx / safe, gy / safe


def _weight(d, tSS):
    return (d * torch.exp(-(d * d) / tSS)) ** 4


def _rgc(I, M, fwhm, tSS=None):
    """CGLH over its sum of weights of [f][H][W] float64 frames, no shift (differentiable in I and
    tSS)."""
    R, t0, _ = _fht_geometry(M, fwhm)
    tSS = torch.tensor(t0, dtype=I.dtype, device=I.device) if tSS is None else tSS
    f, H, W = I.shape
    ux, uy = _unit_field(I)
    pad = (R, R + 1, R, R + 1)
    ux, uy = torch.nn.functional.pad(ux, pad), torch.nn.functional.pad(uy, pad)
    inside = torch.nn.functional.pad(torch.ones(H, W, dtype=I.dtype, device=I.device), pad)
    num, den = torch.zeros_like(I), torch.zeros(H, W, dtype=I.dtype, device=I.device)
    for i, j in _fht_taps(M, fwhm):
        a = ux[:, R + j:R + j + H, R + i:R + i + W]
        b = uy[:, R + j:R + j + H, R + i:R + i + W]
        d = torch.tensor(math.hypot(i, j), dtype=I.dtype, device=I.device)
        w = _weight(d, tSS)
        t = 1 - (b * i - a * j).abs() / d
        num = num + w * torch.where(a * i + b * j < 0, t, torch.zeros_like(t))
        den = den + w * inside[R + j:R + j + H, R + i:R + i + W]
    return num / den


def _cubic(x):
    x = x.abs()
    near = x * x * (1.5 * x - 2.5) + 1
    far = -0.5 * x ** 3 + 2.5 * x * x - 4 * x + 2
    return torch.where(x < 1, near, torch.where(x < 2, far, torch.zeros_like(x)))


def _sample(a, x, y):
    """Catmull-Rom samples of [..., h, w] at positions x, y (broadcast together), bilinear with
    extrapolation where the 4 x 4 support leaves the image."""
    h, w = a.shape[-2:]
    u0, v0 = torch.floor(x).long(), torch.floor(y).long()
    ok = (u0 > 0) & (u0 < w - 2) & (v0 > 0) & (v0 < h - 2)
    q = 0
    for j in range(4):
        v = (v0 - 1 + j).clamp(0, h - 1)
        p = 0
        for i in range(4):
            u = (u0 - 1 + i).clamp(0, w - 1)
            p = p + a[..., v, u] * _cubic(x - (u0 - 1 + i))
        q = q + p * _cubic(y - (v0 - 1 + j))
    xb, yb = x.clamp(0, w - 2).long(), y.clamp(0, h - 2).long()
    xf, yf = x - xb, y - yb
    lo = a[..., yb, xb] + xf * (a[..., yb, xb + 1] - a[..., yb, xb])
    hi = a[..., yb + 1, xb] + xf * (a[..., yb + 1, xb + 1] - a[..., yb + 1, xb])
    return torch.where(ok, q, lo + yf * (hi - lo))


def _rgc_shifted(I, M, fwhm, sx, sy):
    """(CGLH over its sum of weights, intensity) of frames with shifts sx, sy [f] in output pixels."""
    R, tSS, tSO = _fht_geometry(M, fwhm)
    f, H, W = I.shape
    dev = I.device
    ux, uy = _unit_field(I)
    X, Y = torch.arange(W, device=dev).double(), torch.arange(H, device=dev).double()
    cx, cy = X + sx[:, None], Y + sy[:, None]  # [f][W], [f][H]: centres less a half
    bx, by = torch.trunc(cx).long(), torch.trunc(cy).long()
    num, den = torch.zeros_like(I), torch.zeros_like(I)
    fi = torch.arange(f, device=dev)[:, None, None]
    for j in range(-R, R + 2):
        vy = by + j
        for i in range(-R, R + 2):
            vx = bx + i
            dx, dy = (vx - cx)[:, None, :], (vy - cy)[:, :, None]
            d = torch.sqrt(dx * dx + dy * dy)
            ok = (d <= tSO) & (d > 0) & ((vx >= 0) & (vx < W))[:, None, :] & ((vy >= 0) & (vy < H))[:, :, None]
            at = (fi, vy.clamp(0, H - 1)[:, :, None], vx.clamp(0, W - 1)[:, None, :])
            a, b = ux[at], uy[at]
            w = _weight(d, tSS) * ok
            den += w
            t = w * (1 - (b * dx - a * dy).abs() / torch.where(d > 0, d, torch.ones_like(d)))
            num += torch.where(a * dx + b * dy < 0, t, torch.zeros_like(t))
    v = torch.empty_like(I)
    for k in range(f):
        if sx[k] == 0 and sy[k] == 0:
            v[k] = I[k]
        else:
            v[k] = _sample(I[k], cx[k][None, :], cy[k][:, None])
    return num / den, v


class _Cumulants:
    """AVG, VAR, TAC2, INT of a block fed in batches of frames."""

    def __init__(self, n, weighting, twice=False):
        self.n, self.weighting, self.twice, self.last, self.sums = n, weighting, twice, None, None

    def add(self, c, v, sens):
        c = torch.where(c >= 0, c, torch.zeros_like(c)) ** sens
        x = v * c if self.weighting else c
        full = x if self.last is None else torch.cat([self.last[None], x])
        s = [x.sum(0), (x * x).sum(0), (full[1:] * full[:-1]).sum(0), v.sum(0)]
        self.sums = s if self.sums is None else [a + b for a, b in zip(self.sums, s)]
        self.last = x[-1].clone()

    def slices(self):
        n = self.n
        avg = self.sums[0] / n
        tac = self.sums[2] / max(1, n - 1) / (max(1, n - 1) if self.twice else 1) if n > 1 else 0 * avg
        return [torch.nan_to_num(o, nan=0.0) for o in (avg, self.sums[1] / n - avg * avg, tac - avg * avg,
                                                       self.sums[3] / n)]


def _batches(n, pixels, most=4e7):
    step = max(1, int(most / pixels))
    return [(t, min(n, t + step)) for t in range(0, n, step)]


def _exact_fht(case, raw, seed):
    M, n = case["mag"], case["frames"]
    cum = _Cumulants(n, case.get("weighting", True))
    shift = [torch.from_numpy(np.float32(M) * a).to(DEV).double() for a in _shifts(seed, n)] if case["vibration"] else None
    for a, b in _batches(n, case["width"] * case["height"] * M * M):
        I = _interpolate(raw[a:b], M)
        if shift:
            c, v = _rgc_shifted(I, M, case["radius"], shift[0][a:b], shift[1][a:b])
        else:
            c, v = _rgc(I, M, case["radius"]), I
        cum.add(c, v, case["sens"])
    return {k: o[None] for k, o in zip(SLICES, cum.slices())}


def _exact_sweep(case, raw):
    out, n = {}, case["frames"]
    for M in _list(case["mags"], int):
        for r in _list(case["radii"], float):
            C, V = [], []
            for a, b in _batches(n, case["width"] * case["height"] * M * M):
                I = _interpolate(raw[a:b], M)
                C.append(_rgc(I, M, r))
                V.append(I)
            C, V = torch.cat(C), torch.cat(V)
            per = []
            for s in _list(case["senses"], int):
                for t, m in _blocks(n):
                    cum = _Cumulants(m, True)
                    cum.add(C[t:t + m], V[t:t + m], s)
                    per.append(torch.stack(cum.slices()))
            per = torch.stack(per).view(len(_list(case["senses"], int)), -1, 4, *C.shape[1:])
            for i, k in enumerate(SLICES):
                out["M%d r%g %s" % (M, r, k)] = per[:, :, i]
    return out


def _twice(g):
    """2x resampling of gradient images [...][h][w]."""
    h, w = g.shape[-2:]
    x = torch.arange(2 * w, device=g.device).double() / 2
    y = torch.arange(2 * h, device=g.device).double() / 2
    return _sample(g, x[None, :], y[:, None])


def _mp_correct(o, M, is3d):
    """Divides a cumulant by its mean over the cells of every sub-pixel phase."""
    z = M if is3d else 1
    P, H, W = o.shape
    b = o.reshape(P // z, z, H // M, M, W // M, M)
    return (b / b.mean(dim=(0, 2, 4), keepdim=True)).reshape(P, H, W)


def _slab(u, x0, y0, w, h):
    """u [...][H2][W2] at columns x0 + 2 q, rows y0 + 2 p; zero where a tap may not read (node 0 and
    beyond the last node)."""
    H2, W2 = u.shape[-2:]
    x = torch.arange(w, device=u.device) * 2 + x0
    y = torch.arange(h, device=u.device) * 2 + y0
    ok = ((y > 0) & (y < H2))[:, None] & ((x > 0) & (x < W2))[None, :]
    return u[..., y.clamp(0, H2 - 1)[:, None], x.clamp(0, W2 - 1)[None, :]] * ok, ok


def _at_nodes(gx, gy, *more):
    """Gradient components as the taps of a node read them: x component of the row above, y component
    of the column to the left, the others of both."""
    up = _before(gx.shape[-2], gx.device)
    left = _before(gx.shape[-1], gx.device)
    return [gx[..., up, :], gy[..., left]] + [g[..., up, :][..., left] for g in more]


def _exact_bic(case, raw):
    M, n, h, w = case["mag"], case["frames"], case["height"], case["width"]
    _, tSS, _ = _bic_geometry(case["radius"])
    cum = _Cumulants(n, True, twice=True)
    for a, b in _batches(n, w * h * M * M):
        f = raw[a:b]
        gx = _twice(f - f[:, :, _before(w, DEV)])
        gy = _twice(f - f[:, _before(h, DEV)])
        gx, gy = _at_nodes(gx, gy)
        m = torch.sqrt(gx * gx + gy * gy)
        m = torch.where(m > 0, m, torch.ones_like(m))
        ux, uy = gx / m, gy / m
        C = torch.empty(b - a, h * M, w * M, dtype=torch.float64, device=DEV)
        for py in range(M):
            for px in range(M):
                num, den = 0, 0
                for nx, ny, dx, dy in _bic_taps(M, case["radius"], px, py):
                    d = math.hypot(dx, dy)
                    if d < 1e-9:
                        continue
                    wt = (d * math.exp(-(d * d) / tSS)) ** 4
                    (p, ok), (q, _) = _slab(ux, nx, ny, w, h), _slab(uy, nx, ny, w, h)
                    t = wt * (1 - (q * dx - p * dy).abs() / d)
                    num = num + torch.where(p * dx + q * dy < 0, t, torch.zeros_like(t))
                    den = den + wt * ok
                C[:, py::M, px::M] = num / den
        x = torch.arange(w * M, device=DEV).double() / M - 0.5
        y = torch.arange(h * M, device=DEV).double() / M - 0.5
        cum.add(C, _sample(f, x[None, :], y[:, None]), case["sens"])
    o = [s[None] for s in cum.slices()]
    return dict(zip(SLICES, [_mp_correct(s, M, False) for s in o[:3]] + o[3:]))


def _exact_mfm(case, cam):
    M, n, h, w, P = case["mag"], case["frames"], case["height"], case["width"], 9
    radius, tSS, tSO = _bic_geometry(case["radius"])
    k0, k1 = -int(radius), int(radius) + 1
    cal = _calibration()
    cum = _Cumulants(n, True)
    X = torch.arange(w, device=DEV).double()[None, :] - (w - 1) / 2
    Y = torch.arange(h, device=DEV).double()[:, None] - (h - 1) / 2
    for a, b in _batches(n, P * w * h * M ** 3):
        f = torch.empty(b - a, P, h, w, dtype=torch.float64, device=DEV)
        for z, r in enumerate(ROI):
            t = cam[a:b, (r // 3) * h:(r // 3 + 1) * h, (r % 3) * w:(r % 3 + 1) * w]
            t = (t - 90.0) / float(cal["Intensity scaling"][z])
            th = -math.radians(float(cal["Theta (degrees)"][z]))
            c, s = math.cos(th), math.sin(th)
            f[:, z] = _sample(t, X * c - Y * s + (w - 1) / 2 - float(cal["X-shift (pixels)"][z]),
                              X * s + Y * c + (h - 1) / 2 - float(cal["Y-shift (pixels)"][z]))
        g = _at_nodes(_twice(f - f[..., _before(w, DEV)]), _twice(f - f[..., _before(h, DEV), :]),
                      _twice(f - f[:, _before(P, DEV)]))
        m = torch.sqrt(sum(c * c for c in g))
        m = torch.where(m > 0, m, torch.ones_like(m))
        u = [c / m for c in g]
        C = torch.empty(b - a, P * M, h * M, w * M, dtype=torch.float64, device=DEV)
        V = torch.empty_like(C)
        x = torch.arange(w * M, device=DEV).double() / M - 0.5
        y = torch.arange(h * M, device=DEV).double() / M - 0.5
        lateral = _sample(f, x[None, :], y[:, None])
        for zM in range(P * M):
            zc = (zM + 0.5) / M
            z0 = 0 if zc < 0.5 else P - 2 if zc - 0.5 >= P - 1 else int(math.floor(zc - 0.5 + 1e-9))
            v_1, v0, v1 = lateral[:, max(z0 - 1, 0)], lateral[:, z0], lateral[:, z0 + 1]
            v2 = lateral[:, min(z0 + 1, P - 1)]
            t = zc - (z0 + 0.5)
            V[:, zM] = (-0.5 * v_1 + 1.5 * v0 - 1.5 * v1 + 0.5 * v2) * t ** 3 + \
                (v_1 - 2.5 * v0 + 2 * v1 - 0.5 * v2) * t * t + (-0.5 * v_1 + 0.5 * v1) * t + v0
        r0, r1 = -int(2 * radius), int(2 * radius + 1)
        z = torch.arange(P, device=DEV)
        for py in range(M):
            for px in range(M):
                xc, yc = (px + 0.5) / M, (py + 0.5) / M
                kx, ky = int(2 * xc + 1e-9), int(2 * yc + 1e-9)
                num = [0] * M
                den = [0] * M
                for j in range(r0, r1 + 1):
                    for i in range(r0, r1 + 1):
                        dx, dy = (kx + i) / 2 - xc, (ky + j) / 2 - yc
                        if dx * dx + dy * dy > tSO * tSO:
                            continue
                        s = [_slab(c, kx + i, ky + j, w, h) for c in u]
                        ok2, s = s[0][1], [v[0] for v in s]
                        for k in range(k0, k1 + 1):
                            okz = (z + k > 0) & (z + k < P)
                            at = (z + k).clamp(0, P - 1)
                            gx, gy, gz = [c[:, at] * okz[:, None, None] for c in s]
                            for pz in range(M):
                                dz = k - (pz + 0.5) / M
                                d = math.sqrt(dx * dx + dy * dy + dz * dz)
                                if d < 1e-9 or d > tSO:
                                    continue
                                wt = (d * math.exp(-(d * d) / tSS)) ** 4
                                cr = torch.sqrt((dy * gz - dz * gy) ** 2 + (dz * gx - dx * gz) ** 2 +
                                                (dx * gy - dy * gx) ** 2)
                                t = wt * (1 - cr / d)
                                num[pz] = num[pz] + torch.where(gx * dx + gy * dy + gz * dz < 0, t,
                                                                torch.zeros_like(t))
                                den[pz] = den[pz] + wt * (okz[:, None, None] & ok2)
                for pz in range(M):
                    C[:, pz::M, py::M, px::M] = num[pz] / den[pz]
        cum.add(C, V, case["sens"])
    o = cum.slices()
    return dict(zip(SLICES, [_mp_correct(s, M, True) for s in o[:3]] + o[3:]))


def _exact_adjoint(case, raw):
    n, h, w, M = case["frames"], case["height"], case["width"], case["mag"]
    fwhm = torch.tensor(float(np.float32(case["radius"])), dtype=torch.float64, device=DEV, requires_grad=True)
    S = torch.tensor(float(np.float32(case["sens"])), dtype=torch.float64, device=DEV, requires_grad=True)
    sb = torch.tensor(float(np.float32(case["sigma"])), dtype=torch.float64, device=DEV, requires_grad=True)

    def frame_term(x):
        sigma = fwhm / float(np.float32(2.354))
        I = _interpolate(x, M)
        c = _rgc(I, M, case["radius"], 2 * sigma * sigma * M * M)
        pos = c > 0
        return (I * torch.where(pos, torch.where(pos, c, torch.ones_like(c)) ** S, torch.zeros_like(c))).sum(0) / n

    with torch.no_grad():
        R = sum(frame_term(raw[t:t + 1]) for t in range(n))
    R.requires_grad_(True)
    mean = raw.mean(0).requires_grad_(True)
    r = math.ceil(4 * float(sb))
    u = torch.arange(-r, r + 1, device=DEV).double()
    k = torch.exp(-u * u / (2 * sb * sb))
    k = k / k.sum()
    B = torch.nn.functional.conv2d(R[None, None], k[None, None, None, :], padding=(0, r))
    B = torch.nn.functional.conv2d(B, k[None, None, :, None], padding=(r, 0))[0, 0]
    D = B.reshape(h, M, w, M).mean(dim=(1, 3))
    d, f = D.detach(), mean.detach()
    alpha = ((d - d.mean()) * (f - f.mean())).sum() / ((d - d.mean()) ** 2).sum()
    loss = ((alpha * D + (f.mean() - alpha * d.mean()) - mean) ** 2).mean()
    loss.backward()
    out = torch.empty_like(raw)
    for t in range(n):
        x = raw[t:t + 1].clone().requires_grad_(True)
        frame_term(x).backward(R.grad)
        out[t] = x.grad[0] + mean.grad / n
    return {"loss": float(loss), "fwhm": float(fwhm.grad), "S": float(S.grad), "sigma": float(sb.grad), "frames": out}


def _exact_shifts(raw):
    n, H, W = raw.shape
    R = max(1, min(31, (min(W, H) - 1) // 2))
    F = torch.fft.fft2(raw[0] - raw[0].mean())
    full = torch.fft.ifft2(F.conj() * torch.fft.fft2(raw)).real
    lag = torch.arange(-R, R + 1, device=DEV)
    m = full[:, (lag % H)[:, None], (lag % W)[None, :]].cpu().numpy()
    X, Y = np.meshgrid([-1.0, 0.0, 1.0], [-1.0, 0.0, 1.0])
    sx, sy = np.empty(n), np.empty(n)
    for t in range(n):
        py, px = divmod(int(np.argmax(m[t])), 2 * R + 1)
        ox = oy = 0.0
        if 0 < px < 2 * R and 0 < py < 2 * R:
            v = m[t][py - 1:py + 2, px - 1:px + 2]
            b, c, e = (X * v).sum() / 6, (Y * v).sum() / 6, (X * Y * v).sum() / 4
            p, q = (X * X * v).sum() / 2 - v.sum() / 3, (Y * Y * v).sum() / 2 - v.sum() / 3
            det = 4 * p * q - e * e
            if det != 0:
                ox = min(1.0, max(-1.0, (-2 * q * b + e * c) / det))
                oy = min(1.0, max(-1.0, (-2 * p * c + e * b) / det))
        sx[t], sy[t] = px - R + ox, py - R + oy
    return {"x": sx, "y": sy}


def exact(case, seed):
    raw = _frames(case, seed).double()
    kind = case["kind"]
    if kind == "shifts":
        return _exact_shifts(raw)
    if kind == "adjoint":
        return _exact_adjoint(case, raw) if _taps_done(case) < 2.5e10 else None
    with torch.no_grad():
        if kind == "fht":
            return _exact_fht(case, raw, seed) if not case["vibration"] or _taps_done(case) < 4e10 else None
        if kind == "sweep":
            return _exact_sweep(case, raw)
        if kind == "bic":
            return _exact_bic(case, raw)
        return _exact_mfm(case, raw) if _taps_done(case) < 8e10 else None
