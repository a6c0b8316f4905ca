"""Performance cases of the framework's public entry points.

Each case is a dict of plain values; `prepare` makes the inputs and plans a
user's program would hold on the GPU, `run` is one pass through the public
calls, `exact` the same outputs in 64-bit torch arithmetic.  The listed cases
cover the dense transforms (1D rows, 3D volumes, 2D real images with their
gradient, uneven batches, lengths beyond one CTA) and the caller operations
(STFT, CZT, 1D / 3D NUFFT); `draw` gives more of the same ranges: odd, prime
and ragged sizes, both precisions, every transform kind.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import apollofft_b200 as afc
from apollofft_b200 import autograd, workloads
from apollofft_b200.czt import CztPlan
from apollofft_b200.nufft import NufftPlan1D, NufftPlan3D
from apollofft_b200.stft import StftPlan, hann_window

DEV = "cuda:0"


def listed():
    return [
        # one small real volume through the drop-in functions: launch latency and host cost per call
        {"name": "volume_24x32x40_real_f64", "op": "fft3", "dims": "24x32x40", "precision": "f64"},
        # a batch of short signals, forward and inverse, f64 (the plan most callers loop over)
        {"name": "rows_64x4096_c128", "op": "rows", "n": 4096, "batch": 64, "precision": "f64"},
        # the 3D transform of a simulation grid, power of two, f64: the headline configuration
        {"name": "volume_256_c128", "op": "volume", "dims": "256x256x256", "precision": "f64", "kind": "c2c"},
        # a 3D grid of smooth odd lengths in f32
        {"name": "volume_243x250x343_c64", "op": "volume", "dims": "243x250x343", "precision": "f32", "kind": "c2c"},
        # many rows at once in f32 (a spectrogram-sized batch): bandwidth of one pass
        {"name": "rows_16384x4096_c64", "op": "rows", "n": 4096, "batch": 16384, "precision": "f32"},
        # long signals, several passes over memory
        {"name": "rows_8x1048576_c64", "op": "rows", "n": 1048576, "batch": 8, "precision": "f32"},
        # signals of every length at once: powers of two, 7-smooth lengths, primes
        {"name": "uneven_4096_c64", "op": "uneven", "count": 4096, "lo": 64, "hi": 65536, "precision": "f32"},
        # training through a spectral loss: real images, forward and gradient
        {"name": "images_8x2048x2048_grad_f32", "op": "images", "batch": 8, "h": 2048, "w": 2048, "half": False,
         "precision": "f32"},
        # audio analysis and resynthesis
        {"name": "stft_4194304_1024_256_f64", "op": "stft", "n": 4194304, "frame": 1024, "hop": 256,
         "precision": "f64"},
        # zoomed spectra of many records
        {"name": "czt_4096x1000_f64", "op": "czt", "lanes": 4096, "n": 1000, "m": 1000, "precision": "f64"},
        # non-uniform samples to a spectrum and back, 1D
        {"name": "nufft1d_65536_1048576", "op": "nufft1d", "n": 65536, "points": 1048576, "width": 6,
         "layout": "uniform"},
        # gridding of a 3D acquisition and its adjoint direction
        {"name": "nufft3d_64_262144", "op": "nufft3d", "dims": "64x64x64", "points": 262144, "width": 6,
         "layout": "uniform"},
    ]


# ── drawn cases ──

def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _smooth_below(v):
    """The largest 2^a 3^b 5^c 7^d <= v."""
    s = workloads._smooth7(v)
    return s[-1]


def _length(rng, lo, hi):
    """A power of two, a 7-smooth length, or whatever comes (odd, prime, ...)."""
    v = _log(rng, lo, hi)
    k = rng.randrange(3)
    if k == 0:
        return max(lo, 1 << int(round(math.log2(v))) if 1 << int(round(math.log2(v))) <= hi else v)
    if k == 1:
        return max(lo, _smooth_below(v))
    return v


def _axis(rng, lo, hi):
    """Length of an axis that is not the last: any up to 256, powers of two
    above (where grids and image heights are powers of two in practice)."""
    v = _length(rng, lo, hi)
    return v if v <= 256 else 1 << int(math.log2(v))


def draw(rng):
    op = rng.choice(["fft3", "rows", "rows", "volume", "volume", "uneven", "images", "stft", "czt", "nufft1d",
                     "nufft3d"])
    prec = rng.choice(["f32", "f64"])
    if op == "fft3":
        return {"op": op, "dims": "x".join(str(rng.randint(8, 48)) for _ in range(3)), "precision": prec}
    if op == "rows":
        n = _length(rng, 64, 1 << 20)
        # lengths without a small factorization take a convolution of two to four times the length
        total = 1 << rng.randint(17, 25 if prec == "f32" else 24)
        if _smooth_below(n) != n:
            total = min(total, 1 << 22)
        if n & (n - 1) == 0 and n <= 4096 and rng.randrange(3) == 0:
            prec = rng.choice(["tc_fp16", "tc_bf16"])
        return {"op": op, "n": n, "batch": max(2, total // n), "precision": prec}
    if op == "volume":
        while True:
            d = [_axis(rng, 16, 384), _axis(rng, 16, 384), _length(rng, 16, 384)]
            if d[0] * d[1] * d[2] <= 1 << 24:
                break
        kind = rng.choice(["c2c", "c2c", "r2c_full", "r2c_half"])
        if kind == "r2c_half":
            d[2] = _smooth_below(d[2])  # half spectra are planned for smooth last axes
        return {"op": op, "dims": "x".join(map(str, d)), "precision": prec, "kind": kind}
    if op == "uneven":
        return {"op": op, "count": _log(rng, 64, 2048), "lo": 64, "hi": _log(rng, 2048, 65536), "precision": prec}
    if op == "images":
        h, w = _axis(rng, 128, 2048), _length(rng, 128, 2048)
        half = rng.randrange(2) == 1
        if half:
            w = _smooth_below(w)
        return {"op": op, "batch": max(1, min(8, (1 << 24) // (h * w))), "h": h, "w": w, "half": half,
                "precision": prec}
    if op == "stft":
        frame = _length(rng, 64, 4096)
        return {"op": op, "n": _log(rng, 1 << 16, 1 << 22), "frame": frame,
                "hop": max(1, frame // rng.choice([2, 3, 4])), "precision": prec}
    if op == "czt":
        return {"op": op, "lanes": _log(rng, 64, 4096), "n": _log(rng, 64, 1000), "m": _log(rng, 64, 1000),
                "precision": prec}
    if op == "nufft1d":
        return {"op": op, "n": _length(rng, 1024, 65536), "points": _log(rng, 1 << 14, 1 << 20),
                "width": rng.randint(4, 8), "layout": rng.choice(["uniform", "dense"])}
    layout = rng.choice(["uniform", "dense"])
    return {"op": op, "dims": "x".join(str(rng.randint(16, 64)) for _ in range(3)),
            "points": _log(rng, 1 << 13, 1 << (14 if layout == "dense" else 17)), "width": rng.randint(4, 7),
            "layout": layout}


# ── inputs ──

def _dims(case):
    return [int(v) for v in case["dims"].split("x")]


def _real_t(case):
    return torch.float64 if case["precision"] == "f64" else torch.float32


def _cplx_t(case):
    return torch.complex128 if case["precision"] == "f64" else torch.complex64


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _normal(shape, dtype, g):
    return torch.randn(shape, dtype=dtype, device=DEV, generator=g)


def _uniform(shape, dtype, g):
    """Uniform in [-1, 1), real and imaginary parts for complex types."""
    if dtype.is_complex:
        rt = torch.float64 if dtype == torch.complex128 else torch.float32
        return torch.complex(_uniform(shape, rt, g), _uniform(shape, rt, g))
    return torch.rand(shape, dtype=dtype, device=DEV, generator=g) * 2 - 1


def _points(count, length, layout, g):
    """Sample positions over [0, length): uniform, or dense around the middle
    (a trajectory through the centre samples it far more often)."""
    u = torch.rand(count, dtype=torch.float64, device=DEV, generator=g)
    if layout == "dense":
        v = torch.rand(count, dtype=torch.float64, device=DEV, generator=g)
        u = 0.5 + (u - 0.5) * v * v
    return u * length


def _inputs(case, seed):
    """Input tensors of a case, from the seed alone."""
    g = _gen(seed)
    op = case["op"]
    if op == "fft3":
        return {"x": _normal(_dims(case), _real_t(case), g)}
    if op == "rows":
        return {"x": _uniform((case["batch"], case["n"]), _cplx_t(case), g)}
    if op == "volume":
        dt = _cplx_t(case) if case["kind"] == "c2c" else _real_t(case)
        return {"x": _normal(_dims(case), dt, g)}
    if op == "uneven":
        lens = _lengths(case)
        return {"x": _uniform((int(lens.sum()),), _cplx_t(case), g)}
    if op == "images":
        h, w = case["h"], case["w"]
        x = _normal((case["batch"], h, w), _real_t(case), g)
        fy = torch.fft.fftfreq(h, device=DEV, dtype=torch.float64)[:, None]
        fx = (torch.fft.rfftfreq(w, device=DEV, dtype=torch.float64) if case["half"]
              else torch.fft.fftfreq(w, device=DEV, dtype=torch.float64))[None, :]
        weight = 1.3 * torch.exp(-8.0 * torch.sqrt(fy * fy + fx * fx)) + 0.1
        return {"x": x, "weight2": (2 * weight * weight).to(_real_t(case))}
    if op == "stft":
        return {"x": _uniform((case["n"],), _real_t(case), g)}
    if op == "czt":
        return {"x": _uniform((case["lanes"], case["n"]), _cplx_t(case), g)}
    if op == "nufft1d":
        return {"pos": _points(case["points"], float(case["n"]) * 0.5, case["layout"], g),
                "val": _normal((case["points"],), torch.complex128, g),
                "coef": _normal((case["n"],), torch.complex128, g)}
    d = _dims(case)
    pos = torch.stack([_points(case["points"], float(n) * 0.5, case["layout"], g) for n in d], dim=1).contiguous()
    return {"pos": pos, "val": _normal((case["points"],), torch.complex128, g),
            "coef": _normal(d, torch.complex128, g)}


def _lengths(case):
    return workloads.c3_lengths(case["count"], case["lo"], case["hi"])


def _czt_params(case):
    """An arc of the unit circle: one eighth of the band around its middle."""
    m = case["m"]
    return np.exp(2j * np.pi * 0.1875), np.exp(-2j * np.pi * 0.125 / m)


def prepare(case, seed):
    st = dict(_inputs(case, seed))
    st["case"] = case
    op = case["op"]
    if op == "rows":
        st["plan"] = afc.CudaPlan([case["n"]], precision=case["precision"], batch=case["batch"])
    elif op == "volume":
        st["plan"] = afc.CudaPlan(_dims(case), precision=case["precision"], kind=case["kind"])
    elif op == "uneven":
        st["plan"] = afc.BatchPlan(_lengths(case), precision=case["precision"])
        st["out"] = torch.empty_like(st["x"])
    elif op == "images":
        st["x"].requires_grad_(True)
    elif op == "stft":
        st["plan"] = StftPlan(case["frame"], case["hop"], precision=case["precision"])
    elif op == "czt":
        a, w = _czt_params(case)
        st["plan"] = CztPlan(case["n"], case["m"], a, w, precision=case["precision"])
    elif op == "nufft1d":
        st["plan"] = NufftPlan1D(case["n"], 0.5, kernel_width=case["width"])
    elif op == "nufft3d":
        st["plan"] = NufftPlan3D(_dims(case), (0.5, 0.5, 0.5), kernel_width=case["width"])
    return st


# ── one pass ──

def run(st):
    case = st["case"]
    op = case["op"]
    if op == "fft3":
        prec = "high_accuracy" if case["precision"] == "f64" else "low_precision"
        y = afc.fft3(st["x"], prec)
        return y, afc.ifft3(y, prec)
    if op in ("rows", "volume"):
        y = st["plan"].execute(st["x"])
        return y, st["plan"].execute(y, inverse=True)
    if op == "uneven":
        return st["plan"].execute(st["x"], out=st["out"])
    if op == "images":
        # d/dx of sum |weight X|^2: the cotangent of X is 2 weight^2 X
        y = autograd.rfft2(st["x"], half=case["half"])
        gx, = torch.autograd.grad(y, st["x"], y.detach() * st["weight2"])
        return y.detach(), gx
    if op == "stft":
        s = st["plan"].forward(st["x"])
        return s, st["plan"].inverse(s, case["n"])
    if op == "czt":
        return st["plan"].forward(st["x"])
    return st["plan"].type1(st["pos"], st["val"]), st["plan"].type2(st["coef"], st["pos"])


# ── the work a pass cannot do without ──

def _fft_flops(n_total, length):
    return 5.0 * n_total * math.log2(max(2, length))


def work(case):
    op = case["op"]
    csz = 16 if case.get("precision", "f64") == "f64" else 8
    if op in ("fft3", "volume"):
        n = math.prod(_dims(case))
        kind = case.get("kind", "r2c_full")
        spec = n
        if kind == "r2c_half":
            d = _dims(case)
            spec = n // d[2] * (d[2] // 2 + 1)
        one_in = n * csz if kind == "c2c" else n * csz // 2
        f = _fft_flops(n, n) * (1.0 if kind == "c2c" else 0.5)
        return {"bytes": 2.0 * (one_in + spec * csz), "flops": 2 * f}
    if op == "rows":
        n = case["n"] * case["batch"]
        return {"bytes": 4.0 * n * csz, "flops": 2 * _fft_flops(n, case["n"])}
    if op == "uneven":
        lens = _lengths(case).astype(np.float64)
        return {"bytes": 2.0 * csz * float(lens.sum()), "flops": 5.0 * float((lens * np.log2(lens)).sum())}
    if op == "images":
        n = case["batch"] * case["h"] * case["w"]
        spec = case["batch"] * case["h"] * (case["w"] // 2 + 1) if case["half"] else n
        # forward: image in, spectrum out; cotangent: spectrum in and out; adjoint: cotangent in, gradient out
        return {"bytes": 2.0 * (n * csz // 2) + 4.0 * spec * csz, "flops": _fft_flops(n, case["h"] * case["w"])}
    if op == "stft":
        frames = 1 + -(-case["n"] // case["hop"])
        spec = frames * case["frame"]
        return {"bytes": 2.0 * case["n"] * csz // 2 + 2.0 * spec * csz, "flops": 1.0 * _fft_flops(spec, case["frame"])}
    if op == "czt":
        lanes, n, m = case["lanes"], case["n"], case["m"]
        ln = 1 << (n + m - 2).bit_length()
        return {"bytes": float(csz) * lanes * (n + m), "flops": 2 * _fft_flops(lanes * ln, ln)}
    if op == "nufft1d":
        n, p, t = case["n"], case["points"], 2 * case["width"] + 1
        return {"bytes": 2.0 * (24 * p + 16 * n), "flops": 2 * (4.0 * t * p + _fft_flops(2 * n, 2 * n))}
    d, p, t = _dims(case), case["points"], 2 * case["width"] + 1
    n, m = math.prod(d), math.prod(1 << (2 * v - 1).bit_length() for v in d)
    return {"bytes": 2.0 * (40 * p + 16 * n), "flops": 2 * (4.0 * t ** 3 * p + _fft_flops(m, m))}


# ── accuracy ──

def tolerance(case):
    # about four times the largest distance from the 64-bit result measured
    # over the listed and drawn sizes of each precision
    op = case["op"]
    prec = case.get("precision", "f64")
    if op in ("nufft1d", "nufft3d"):
        return {"rel": 1e-12}  # both directions sum in f64; order of the sums differs
    if prec == "tc_bf16":
        return {"rel": 3e-5}
    if prec == "tc_fp16":
        return {"rel": 4e-6}
    if op == "czt":
        return {"rel": 1e-12 if prec == "f64" else 4e-6}
    return {"rel": 5e-15 if prec == "f64" else 2e-6}


def _exact_nufft(case, seed):
    st = _inputs(case, seed)
    pos, val, coef = st["pos"], st["val"], st["coef"]
    two_pi = 2.0 * math.pi

    def phases(x, length, ks):  # exp(-2 pi i k x / length), the turn reduced before the angle
        turn = x[:, None] / length * ks[None, :]
        return torch.polar(torch.ones_like(turn), -two_pi * (turn - torch.round(turn)))

    def signed(n):
        k = torch.arange(n, device=DEV, dtype=torch.float64)
        return torch.where(k <= n // 2, k, k - n)

    p = pos.shape[0]
    if case["op"] == "nufft1d":
        n = case["n"]
        length = n * 0.5
        # k = 256 a + b, both signs: the sum factors into a product of two small tables
        na = -(-n // 256) + 1
        a0 = -(n // 2) // 256 - 1
        ka = 256.0 * (torch.arange(na + 2, device=DEV, dtype=torch.float64) + a0)
        kb = torch.arange(256, device=DEV, dtype=torch.float64)
        idx = (signed(n) - 256.0 * a0).long()
        table = torch.zeros(((na + 2) * 256,), dtype=torch.complex128, device=DEV)
        coef_t = table.clone()
        coef_t[idx] = coef
        out2 = torch.empty(p, dtype=torch.complex128, device=DEV)
        acc = table.view(na + 2, 256)
        for s in range(0, p, 1 << 16):
            e = slice(s, s + (1 << 16))
            ea, eb = phases(pos[e], length, ka), phases(pos[e], length, kb)
            acc += (ea * val[e][:, None]).T @ eb
            out2[e] = ((eb.conj() @ coef_t.view(na + 2, 256).T) * ea.conj()).sum(1)
        return acc.reshape(-1)[idx], out2
    d = _dims(case)
    m = math.prod(1 << (max(2 * v, 2 * case["width"] + 1) - 1).bit_length() for v in d)
    f = torch.zeros((d[0], d[1] * d[2]), dtype=torch.complex128, device=DEV)
    out2 = torch.empty(p, dtype=torch.complex128, device=DEV)
    step = 1 << 14
    for s in range(0, p, step):
        e = slice(s, s + step)
        ex, ey, ez = (phases(pos[e, i].contiguous(), d[i] * 0.5, signed(d[i])) for i in range(3))
        eyz = (ey[:, :, None] * ez[:, None, :]).reshape(ex.shape[0], -1)
        f += (ex * val[e][:, None]).T @ eyz
        out2[e] = ((eyz.conj() @ coef.reshape(d[0], -1).T) * ex.conj()).sum(1)
    return f.reshape(d), out2 / m  # the plan's inverse axis passes are normalized


def exact(case, seed):
    op = case["op"]
    if op in ("nufft1d", "nufft3d"):
        return _exact_nufft(case, seed)
    st = _inputs(case, seed)
    x = st["x"].to(torch.complex128)
    if op == "fft3":
        return torch.fft.fftn(x), x.real
    if op == "rows":
        return torch.fft.fft(x), x
    if op == "volume":
        if case["kind"] == "c2c":
            return torch.fft.fftn(x), x
        y = torch.fft.fftn(x) if case["kind"] == "r2c_full" else torch.fft.rfftn(x.real)
        return y, x.real
    if op == "uneven":
        h = x.cpu().numpy()
        out, o = np.empty_like(h), 0
        for n in _lengths(case):
            out[o:o + n] = np.fft.fft(h[o:o + n])
            o += int(n)
        return out
    if op == "images":
        w2 = st["weight2"].to(torch.float64)
        y = torch.fft.rfft2(x.real) if case["half"] else torch.fft.fft2(x)
        g = y * w2
        if case["half"]:
            full = torch.zeros(x.shape, dtype=torch.complex128, device=DEV)
            full[..., : g.shape[-1]] = g
            g = full
        return y, torch.fft.ifft2(g).real * (case["h"] * case["w"])
    if op == "stft":
        frame, hop, n = case["frame"], case["hop"], case["n"]
        frames = 1 + -(-n // hop)
        # the analysis window as the plan holds it, in the plan's precision
        win = torch.from_numpy(hann_window(frame)).to(DEV, _real_t(case)).to(torch.float64)
        half = frame // 2
        pad = torch.zeros((frames - 1) * hop + frame, dtype=torch.float64, device=DEV)
        keep = min(n, pad.numel() - half)
        pad[half:half + keep] = x.real[:keep]
        fr = pad.unfold(0, frame, hop) * win
        acc, wsum = torch.zeros_like(pad), torch.zeros_like(pad)
        at = (torch.arange(frames, device=DEV) * hop)[:, None] + torch.arange(frame, device=DEV)[None, :]
        acc.index_add_(0, at.reshape(-1), (fr * win).reshape(-1))
        wsum.index_add_(0, at.reshape(-1), (win * win).expand(frames, frame).reshape(-1))
        sig = torch.where(wsum > 0, acc / wsum.clamp_min(1e-300), torch.zeros_like(acc))[half:half + n]
        return torch.fft.fft(fr.to(torch.complex128)), torch.nn.functional.pad(sig, (0, n - sig.numel()))
    n, m = case["n"], case["m"]
    # a = exp(2 pi i 3/16), w = exp(-2 pi i / (8 m)): whole turns taken out in integers
    j = torch.arange(n, device=DEV, dtype=torch.int64)
    k = torch.arange(m, device=DEV, dtype=torch.int64)
    num = (j[:, None] * k[None, :]) * 2 + 3 * m * j[:, None]  # turns: -(num / (16 m))
    ang = (num % (16 * m)).to(torch.float64) / (16.0 * m)
    return x @ torch.polar(torch.ones_like(ang), -2.0 * math.pi * ang)
