"""The compile-time power-of-two engine against numpy and against the general
engine (AFC_FX=0 at plan creation) over every form it takes: contiguous and
strided lanes, real and half spectra, mirrored columns, the two passes of long
lengths, convolutions and analysis frames, with lane counts that leave
remainders in its tiles."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {"f64": 1e-13, "f32": 2e-6}  # a few units of rounding times log2 n, well under the parity bars


def rel(a, b):
    a, b = np.asarray(a).ravel(), np.asarray(b).ravel()
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def plans(afc, dims, **kw):
    """(compile-time plan, general plan)"""
    fx = afc.CudaPlan(list(dims), cached=False, **kw)
    os.environ["AFC_FX"] = "0"
    try:
        return fx, afc.CudaPlan(list(dims), cached=False, **kw)
    finally:
        del os.environ["AFC_FX"]


def check(afc, cuda, dims, batch, precision, kind):
    import torch
    rng = np.random.default_rng(sum(dims) + batch)
    shape = (batch,) + tuple(dims)
    x = rng.standard_normal(shape)
    if kind == "c2c":
        x = x + 1j * rng.standard_normal(shape)
    axes = tuple(range(1, len(shape)))
    fx, gen = plans(afc, dims, precision=precision, kind=kind, batch=batch)
    t = torch.from_numpy(x.astype(fx.in_dtype(False))).to(cuda)
    x = t.cpu().numpy().astype(x.dtype)
    ref = np.fft.rfftn(x, axes=axes) if kind == "r2c_half" else np.fft.fftn(x, axes=axes)
    y, yg = fx.execute(t), gen.execute(t)
    tol = TOL[precision]
    assert rel(y.cpu().numpy(), ref) < tol
    assert rel(y.cpu().numpy(), yg.cpu().numpy()) < tol
    b, bg = fx.execute(y, inverse=True), gen.execute(y, inverse=True)
    assert rel(b.cpu().numpy(), x) < tol
    assert rel(b.cpu().numpy(), bg.cpu().numpy()) < tol
    g = torch.from_numpy(ref.astype(fx.out_dtype(False))).to(cuda)
    assert rel(fx.adjoint(g).cpu().numpy(), gen.adjoint(g).cpu().numpy()) < tol
    if kind == "c2c":  # in place
        z = t.clone()
        fx.execute(z, out=z)
        assert torch.equal(z.reshape(-1), y.reshape(-1))


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("kind", ["c2c", "r2c_full", "r2c_half"])
@pytest.mark.parametrize("n,batch", [(64, 1), (64, 33), (128, 17), (256, 9), (512, 5), (1024, 3), (2048, 3), (4096, 2),
                                     (243, 10), (250, 1), (343, 11)])
def test_rows(afc, cuda, precision, kind, n, batch):
    check(afc, cuda, (n,), batch, precision, kind)


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("kind", ["c2c", "r2c_full", "r2c_half"])
@pytest.mark.parametrize("dims", [(64, 1), (64, 2), (64, 3), (128, 7), (256, 18), (512, 33), (1024, 20), (1024, 130),
                                  (64, 256), (3, 128, 10), (256, 3, 9), (128, 64, 66), (243, 18), (250, 343), (343, 40),
                                  (5, 250, 9)])
def test_columns(afc, cuda, precision, kind, dims):
    if kind == "r2c_half" and dims[-1] < 2:
        pytest.skip("a half spectrum needs two points")
    check(afc, cuda, dims, 2, precision, kind)


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("dims,kind", [((8192,), "c2c"), ((16384,), "r2c_full"), ((65536,), "c2c"), ((1 << 20,), "c2c"),
                                       ((16384, 3), "c2c"), ((3, 32768), "r2c_full"), ((24576,), "c2c"),
                                       ((32768,), "r2c_half")])
def test_two_pass_lengths(afc, cuda, precision, dims, kind):
    check(afc, cuda, dims, 3, precision, kind)


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("dims", [(37,), (1031,), (2039,), (4099,), (10007,), (65521,), (1031, 3), (3, 10007)])
@pytest.mark.parametrize("kind", ["c2c", "r2c_full"])
def test_convolution_lengths(afc, cuda, precision, dims, kind):
    check(afc, cuda, dims, 3, precision, kind)


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("n", [64, 128, 256, 512, 1024, 2048, 4096])
def test_caller_operations(afc, cuda, precision, n):
    import torch
    from apollofft_b200.czt import CztPlan
    from apollofft_b200.hilbert import HilbertPlan
    from apollofft_b200.stft import StftPlan
    rng = np.random.default_rng(n)
    rdt = np.float64 if precision == "f64" else np.float32
    cdt = np.complex128 if precision == "f64" else np.complex64
    tol = TOL[precision]
    sig = rng.standard_normal(5 * n + 7).astype(rdt)
    plan = StftPlan(n, n // 4, precision)
    s = plan.forward(torch.from_numpy(sig).to(cuda))
    pad = np.zeros(len(sig) + 3 * n)
    pad[n // 2:n // 2 + len(sig)] = sig
    win = plan.window.astype(rdt).astype(np.float64)
    ref = np.stack([np.fft.fft(pad[m * (n // 4):m * (n // 4) + n] * win) for m in range(s.shape[0])])
    assert rel(s.cpu().numpy(), ref) < tol
    back = plan.inverse(s, len(sig)).cpu().numpy()
    assert rel(back[1:-1], sig[1:-1]) < tol
    x = rng.standard_normal((5, n)).astype(rdt)
    h = HilbertPlan(n, precision).analytic_signal(torch.from_numpy(x).to(cuda)).cpu().numpy()
    mask = np.zeros(n)
    mask[0] = mask[n // 2] = 1
    mask[1:n // 2] = 2
    assert rel(h, np.fft.ifft(np.fft.fft(x.astype(np.float64)) * mask)) < tol
    nin, m = n // 2 - 5, n // 2 + 3  # convolution length n
    z = (rng.standard_normal((3, nin)) + 1j * rng.standard_normal((3, nin))).astype(cdt)
    a, w = np.exp(0.3j), np.exp(-0.7j / m)
    got = CztPlan(nin, m, a, w, precision).forward(torch.from_numpy(z).to(cuda)).cpu().numpy()
    jk = np.outer(np.arange(nin), np.arange(m))
    czt = z.astype(np.complex128) @ np.exp(-0.3j * np.arange(nin)[:, None] - 0.7j / m * jk)
    # the chirps W^(j^2 / 2) carry the rounding of phases up to j^2 / 2
    assert rel(got, czt) < (2e-11 if precision == "f64" else 2e-5)


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("lengths", [
    [8192],                                                       # one transform of two passes
    [65521, 64, 8192, 10007, 1031, 100, 4096, 8192, 16384, 4099],  # every tile kind, general lengths beside them
    [10007] * 5 + [64] * 130 + [128] * 3 + [2048] * 2,             # lanes that leave remainders in a tile
    [100, 210, 997],                                              # nothing for the compile-time engine
])
def test_uneven_batches(afc, cuda, precision, lengths):
    import torch
    rng = np.random.default_rng(len(lengths))
    plan = afc.BatchPlan(lengths, precision=precision)
    cdt = np.complex128 if precision == "f64" else np.complex64
    x = (rng.standard_normal(plan.total) + 1j * rng.standard_normal(plan.total)).astype(cdt)
    t = torch.from_numpy(x).to(cuda)
    for inverse in (False, True):
        f = np.fft.ifft if inverse else np.fft.fft
        ref = np.concatenate([f(x[o:o + n].astype(np.complex128)) for o, n in zip(plan.offsets, plan.lengths)])
        for mode in (0, 0, 1, 2):  # mode 0 twice: direct, then its graph
            out = plan.execute(t, inverse=inverse, mode=mode).cpu().numpy()
            for o, n in zip(plan.offsets, plan.lengths):
                assert rel(out[o:o + n], ref[o:o + n]) < TOL[precision], (mode, int(n))
    z = t.clone()
    plan.execute(z, out=z, mode=2)
    assert torch.equal(z, plan.execute(t, mode=2))


@pytest.mark.parametrize("n", [74, 1031, 8191, 65521, 100003])
def test_chirp_transform_rounding_f32(afc, cuda, n):
    # A level of either FFT rounds an add and a twiddle product, 0.5 u rms each,
    # independent: 0.71 u.  2 log2 M levels, and the chirp before and after, the
    # spectrum product and the narrowed spectrum as four more.  A kernel spectrum
    # computed in FP32 would add log2 M levels of its own.
    m = 1 << (2 * n - 2).bit_length()
    bound = 0.71 * 2.0**-24 * np.sqrt(2 * np.log2(m) + 4)
    rng = np.random.default_rng(n)
    x = (rng.uniform(-1, 1, (4, n)) + 1j * rng.uniform(-1, 1, (4, n))).astype(np.complex64)
    plan = afc.CudaPlan([n], precision="f32", batch=4)
    import torch
    y = plan.execute(torch.from_numpy(x).to(cuda)).cpu().numpy()
    ref = np.fft.fft(x.astype(np.complex128))
    assert np.linalg.norm(y - ref) <= bound * np.linalg.norm(ref)
