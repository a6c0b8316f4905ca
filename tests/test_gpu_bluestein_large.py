"""complex64 Bluestein lengths whose convolution has a complex64 split into two
passes but no complex128 one (of tiles half the points): in a plan of their own
and in an uneven batch, whose tiles have a third of a CTA's shared memory.  The
spectrum of a few impulses is a sum of exponentials with exact integer phases;
random input goes forward and back."""
import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-5  # complex64, as everywhere


def impulses(n):
    """input with a few impulses and its spectrum"""
    x = np.zeros(n, np.complex64)
    ref = np.zeros(n, np.complex128)
    k = np.arange(n, dtype=np.int64)
    for p, a in ((1, 1.0), (n // 3, -0.5 + 0.25j), (n - 2, 0.75j)):
        x[p] += a
        ref += a * np.exp(-2j * np.pi * ((k * p) % n) / n)
    return x, ref


@pytest.mark.parametrize("n", [16777213, 24000001])
def test_single_plan(afc, cuda, n):
    p = afc.CudaPlan([n], precision="f32", cached=False)
    x, ref = impulses(n)
    assert rel_l2(p.execute(torch.from_numpy(x).to(cuda)).cpu().numpy(), ref) < TOL
    r = torch.randn(n, dtype=torch.complex64, device=cuda, generator=torch.Generator(cuda).manual_seed(n))
    back = p.execute(p.execute(r), inverse=True)
    assert float((back - r).norm() / r.norm()) < TOL


def test_uneven_batch(afc, cuda):
    lengths = [64, 2500009, 97, 3000017]
    b = afc.BatchPlan(lengths, precision="f32")
    ins, refs = zip(*(impulses(n) for n in lengths))
    t = torch.from_numpy(np.concatenate(ins)).to(cuda)
    y = b.execute(t)
    back = b.execute(y, inverse=True).cpu().numpy()
    at = 0
    for n, x, ref in zip(lengths, ins, refs):
        assert rel_l2(y[at:at + n].cpu().numpy(), ref) < TOL, n
        assert rel_l2(back[at:at + n], x) < TOL, n
        at += n
