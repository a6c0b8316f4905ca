"""Axes longer than one tensor-map box (256 rows) whose rows are shorter than
128 bytes: every box must start on a 128-byte boundary of shared memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,kind,precision", [
    ((302, 64), "c2c", "f64"), ((875, 128), "r2c_full", "f32"), ((1000, 40), "c2c", "f64"),
    ((1000, 48), "c2c", "f32"), ((1331, 24), "c2c", "f32"), ((343, 30, 32), "r2c_half", "f64"),
    ((257, 18), "c2c", "f64"), ((3000, 16), "c2c", "f32"), ((3, 510, 20), "c2c", "f32"),
])
def test_long_strided_axes(afc, cuda, dims, kind, precision):
    import torch
    rng = np.random.default_rng(7)
    plan = afc.CudaPlan(list(dims), precision=precision, kind=kind)
    x = rng.standard_normal(dims)
    if kind == "c2c":
        x = x + 1j * rng.standard_normal(dims)
    t = torch.from_numpy(x.astype(plan.in_dtype(False))).to(cuda)
    y = plan.execute(t)
    back = plan.execute(y, inverse=True)
    x64 = t.cpu().numpy().astype(x.dtype)
    ref = np.fft.rfftn(x64) if kind == "r2c_half" else np.fft.fftn(x64)
    tol = 1e-12 if precision == "f64" else 1e-5  # the library's parity bars
    got = y.cpu().numpy().reshape(ref.shape)
    assert np.linalg.norm(got - ref) <= tol * np.linalg.norm(ref)
    b = back.cpu().numpy().reshape(dims)
    assert np.linalg.norm(b - x64) <= tol * np.linalg.norm(x64)
