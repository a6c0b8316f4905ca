"""NUFFT spreading and interpolation where the box kernel, its padded weight
rows, its candidate runs and the polynomial kernel can go wrong: every kernel
width, grids one box wide and up, crowded points (a box's points split over
CTAs), points on cell boundaries, against the reference algorithm restated in
numpy; interpolation repeats bit for bit."""
import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle.nufft import RefPlan, RefPlan3, c_type1_1d, c_type1_3d, c_type2_3d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,w,npts,layout", [
    ((16, 16, 16), 2, 500, "uniform"), ((16, 16, 16), 4, 500, "uniform"), ((16, 9, 16), 5, 700, "cells"),
    ((16, 16, 16), 6, 3000, "dense"), ((10, 17, 33), 6, 2500, "uniform"), ((33, 16, 12), 7, 1500, "cells"),
    ((20, 16, 9), 8, 800, "dense"), ((16, 16, 16), 9, 300, "uniform"), ((16, 12, 16), 6, 1, "uniform"),
    ((40, 20, 16), 3, 4000, "dense"),
])
def test_3d_boxes(afc, oracle, cuda, shape, w, npts, layout):
    from apollofft_b200.nufft import NufftPlan3D
    rng = np.random.default_rng(npts + w)
    spacing = (0.5, 0.25, 1.0)
    ref = RefPlan3(shape, spacing, 2, w)
    L = np.array([n * d for n, d in zip(shape, spacing)])
    u = rng.uniform(-0.3, 1.3, (npts, 3))
    if layout == "dense":
        u = 0.5 + 0.03 * rng.standard_normal((npts, 3))
    if layout == "cells":  # on cells and half way between them
        m = np.array(ref.m)
        u = np.round(u * m * 2) / (2 * m)
    pos = np.ascontiguousarray(u * L)
    val = rng.standard_normal(npts) + 1j * rng.standard_normal(npts)
    modes = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    plan = NufftPlan3D(shape, spacing, 2, w)
    p_t = torch.from_numpy(pos).cuda()
    y1 = plan.type1(p_t, torch.from_numpy(val).cuda()).cpu().numpy()
    y2 = plan.type2(torch.from_numpy(modes).cuda(), p_t).cpu().numpy()
    # sums of (2w + 1)^3 rounded products per point
    assert rel_l2(y1, ref.type1(pos, val, oracle)) < 1e-12
    assert rel_l2(y2, ref.type2(modes, pos, oracle)) < 1e-12


@pytest.mark.parametrize("shape,w", [((16, 16, 16), 4), ((16, 10, 13), 5)])
def test_3d_slices(afc, oracle, cuda, shape, w):
    # more points than the box kernels take at a time: their buffers are used again,
    # every slice adds to the grid, the second slice's values go behind the first's
    from apollofft_b200.nufft import NufftPlan3D
    npts = (1 << 18) + 7
    rng = np.random.default_rng(w)
    dx = (1.0, 1.0, 1.0)
    pos = np.ascontiguousarray(rng.uniform(0, 1, (npts, 3)) * np.array(shape))
    val = rng.standard_normal(npts) + 1j * rng.standard_normal(npts)
    modes = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    plan = NufftPlan3D(shape, dx, 2, w)
    p_t = torch.from_numpy(pos).cuda()
    y1 = plan.type1(p_t, torch.from_numpy(val).cuda()).cpu().numpy()
    y2 = plan.type2(torch.from_numpy(modes).cuda(), p_t).cpu().numpy()
    assert rel_l2(y1, c_type1_3d(shape, dx, 2, w, pos, val)) < 1e-12
    assert rel_l2(y2, c_type2_3d(shape, dx, 2, w, modes, pos)) < 1e-12


@pytest.mark.parametrize("shape,w,npts,boxes", [((16, 16, 16), 2, 1024, False), ((16, 16, 16), 2, 1023, True),
                                                ((16, 20, 16), 2, 9000, False), ((16, 16, 16), 3, 3000, True)])
def test_3d_interpolation_line(afc, cuda, shape, w, npts, boxes):
    # boxes take two launches more than tiles (records, sums)
    from apollofft_b200.nufft import NufftPlan3D
    rng = np.random.default_rng(w)
    dx = (1.0, 1.0, 1.0)
    pos = np.ascontiguousarray(rng.uniform(0, 1, (npts, 3)) * np.array(shape))
    modes = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    plan = NufftPlan3D(shape, dx, 2, w)
    m_t, p_t = torch.from_numpy(modes).cuda(), torch.from_numpy(pos).cuda()
    plan.type2(m_t, p_t)
    before = afc.kernel_launch_count()
    y = plan.type2(m_t, p_t).cpu().numpy()
    # placement and three axis passes, bins, offsets, indices, interpolation
    assert afc.kernel_launch_count() - before == (10 if boxes else 8)
    assert rel_l2(y, c_type2_3d(shape, dx, 2, w, modes, pos)) < 1e-12


@pytest.mark.parametrize("n,w,npts", [(1, 2, 5), (3, 6, 40), (64, 4, 1000), (257, 6, 3001), (1000, 8, 500), (50, 13, 64),
                                      (40, 20, 64)])
def test_1d_widths(afc, oracle, cuda, n, w, npts):
    from apollofft_b200.nufft import NufftPlan1D
    rng = np.random.default_rng(n + w)
    ref = RefPlan(n, 0.3, 2, w)
    pos = rng.uniform(-0.5 * n * 0.3, 1.5 * n * 0.3, npts)
    pos[: npts // 4] = np.round(pos[: npts // 4] / 0.15) * 0.15  # on cells
    val = rng.standard_normal(npts) + 1j * rng.standard_normal(npts)
    coef = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    plan = NufftPlan1D(n, 0.3, 2, w)
    p_t = torch.from_numpy(pos).cuda()
    y1 = plan.type1(p_t, torch.from_numpy(val).cuda()).cpu().numpy()
    y2 = plan.type2(torch.from_numpy(coef).cuda(), p_t).cpu().numpy()
    assert rel_l2(y1, ref.type1(pos, val, oracle)) < 1e-12
    assert rel_l2(y2, ref.type2(coef, pos, oracle)) < 1e-12


@pytest.mark.parametrize("n,w,npts", [(32, 2, 16384), (32, 3, 16384), (32, 4, 4096), (33, 5, 4096), (40, 6, 5001),
                                      (64, 7, 8192), (36, 8, 4097), (32, 9, 4099), (48, 12, 5000), (32, 12, 131),
                                      (70000, 8, 430_000)])
def test_1d_sorted(afc, oracle, cuda, n, w, npts):
    # the widths with kernels of their own (4 .. 8) and any other, a window that
    # wraps a grid of two windows, a partly filled warp, bins of more than eight
    # cells (the last case); the case of 131 points is spread unsorted
    from apollofft_b200.nufft import NufftPlan1D
    rng = np.random.default_rng(n + w)
    length = 0.3 * n
    pos = rng.uniform(-0.2, 1.2, npts) * length
    pos[: npts // 4] = 0.01 * length * rng.standard_normal(npts // 4)  # crowded about the wrap
    val = rng.standard_normal(npts) + 1j * rng.standard_normal(npts)
    y = NufftPlan1D(n, 0.3, 2, w).type1(torch.from_numpy(pos).cuda(), torch.from_numpy(val).cuda()).cpu().numpy()
    assert rel_l2(y, c_type1_1d(n, 0.3, 2, w, pos, val)) < 1e-12


@pytest.mark.parametrize("n,w,npts,sort", [
    (1024, 2, 1 << 20, False), (128, 2, 1 << 16, True), (128, 2, (1 << 16) - 1, False), (1024, 3, 1 << 15, True),
    (65536, 3, 1 << 20, False),
    (1024, 4, 1 << 15, True), (1024, 4, (1 << 15) - 1, False), (65536, 6, 1 << 18, True), (1 << 20, 4, 1 << 20, False)])
def test_1d_sorted_line(afc, cuda, n, w, npts, sort):
    # which spreads sort first: three more launches (bins, offsets, indices)
    from apollofft_b200.nufft import NufftPlan1D
    plan = NufftPlan1D(n, 1.0, 2, w)
    g = torch.Generator(device="cuda").manual_seed(n)
    pos = torch.rand(npts, dtype=torch.float64, device="cuda", generator=g) * n
    val = torch.randn(npts, dtype=torch.complex128, device="cuda", generator=g)

    def launches(k):
        before = afc.kernel_launch_count()
        plan.type1(pos[:k], val[:k])
        return afc.kernel_launch_count() - before

    plan.type1(pos, val)
    assert launches(npts) - launches(1) == (3 if sort else 0)


def test_1d_first_call_captured(afc, cuda):
    # Points enough for a sorted spread, on a plan that has never run: the
    # capture may not allocate, the graph may hold no buffer that a later, larger
    # call moves, and both ways of spreading agree to the rounding of sums of
    # npts (2w + 1) / m products a cell.
    from apollofft_b200.nufft import NufftPlan1D
    n, w, npts = 1024, 6, 200_000  # a one-pass grid transform: it needs no workspace
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    pos = torch.rand(npts, dtype=torch.float64, device="cuda", generator=g) * n
    val = torch.randn(npts, dtype=torch.complex128, device="cuda", generator=g)
    big = torch.rand(3 * npts, dtype=torch.float64, device="cuda", generator=g) * n
    bigv = torch.randn(3 * npts, dtype=torch.complex128, device="cuda", generator=g)
    plan, other = NufftPlan1D(n, 1.0, 2, w), NufftPlan1D(n, 1.0, 2, w)
    other.type1(pos, val)  # kernels are loaded outside a capture
    out = torch.zeros(n, dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.type1(pos, val, out=out)
    plan.type1(big, bigv)
    del other
    for _ in range(2):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert rel_l2(out.cpu().numpy(), plan.type1(pos, val).cpu().numpy()) < 1e-13


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("n,w,npts", [(64, 6, 500), (32, 6, 5000), (32, 5, 5000), (40, 13, 500)])
def test_1d_position_not_finite(afc, cuda, bad, n, w, npts):
    # Its weights are not numbers: no type-1 bin is one then, and of the type-2
    # values only its own is not.  Direct and sorted spreads, wide kernels.
    from apollofft_b200.nufft import NufftPlan1D
    rng = np.random.default_rng(n + w)
    pos = rng.uniform(0, n, npts)
    val, coef = (rng.standard_normal(k) + 1j * rng.standard_normal(k) for k in (npts, n))
    plan = NufftPlan1D(n, 1.0, 2, w)
    c_t, v_t = torch.from_numpy(coef).cuda(), torch.from_numpy(val).cuda()
    good = plan.type2(c_t, torch.from_numpy(pos).cuda()).cpu().numpy()
    pos[npts // 3] = bad
    p_t = torch.from_numpy(pos).cuda()
    assert np.isnan(plan.type1(p_t, v_t).cpu().numpy()).all()
    y2 = plan.type2(c_t, p_t).cpu().numpy()
    assert np.isnan(y2[npts // 3])
    keep = np.arange(npts) != npts // 3
    assert np.array_equal(y2[keep], good[keep])


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("shape,w", [((16, 16, 16), 6), ((8, 16, 4), 6), ((4, 4, 4), 10)])
def test_3d_position_not_finite(afc, cuda, bad, shape, w):
    # box, tile and per-point kernels
    from apollofft_b200.nufft import NufftPlan3D
    rng = np.random.default_rng(w)
    npts = 300
    pos = rng.uniform(0, 1, (npts, 3)) * np.array(shape)
    val = rng.standard_normal(npts) + 1j * rng.standard_normal(npts)
    modes = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    plan = NufftPlan3D(shape, (1.0, 1.0, 1.0), 2, w)
    m_t, v_t = torch.from_numpy(modes).cuda(), torch.from_numpy(val).cuda()
    good = plan.type2(m_t, torch.from_numpy(pos).cuda()).cpu().numpy()
    pos[100, 1] = bad
    p_t = torch.from_numpy(pos).cuda()
    assert np.isnan(plan.type1(p_t, v_t).cpu().numpy()).all()
    y2 = plan.type2(m_t, p_t).cpu().numpy()
    assert np.isnan(y2[100])
    keep = np.arange(npts) != 100
    assert rel_l2(y2[keep], good[keep]) < 1e-13


@pytest.mark.parametrize("shape,w,npts", [((16, 16, 16), 6, 20000), ((20, 16, 12), 9, 3000), ((8, 8, 8), 6, 3000),
                                          ((4, 4, 4), 10, 500)])
def test_3d_interpolation_repeats(afc, cuda, shape, w, npts):
    # whatever order the boxes run in and the points were sorted in
    from apollofft_b200.nufft import NufftPlan3D
    g = torch.Generator(device="cuda").manual_seed(npts)
    pos = torch.rand(npts, 3, dtype=torch.float64, device="cuda", generator=g)
    pos = (pos * torch.tensor(shape, dtype=torch.float64, device="cuda")).contiguous()
    modes = torch.randn(shape, dtype=torch.complex128, device="cuda", generator=g)
    plan = NufftPlan3D(shape, (1.0, 1.0, 1.0), 2, w)
    first = plan.type2(modes, pos)
    for _ in range(5):
        assert torch.equal(torch.view_as_real(plan.type2(modes, pos)), torch.view_as_real(first))
    swap = torch.randperm(npts, device="cuda", generator=g)
    assert torch.equal(torch.view_as_real(plan.type2(modes, pos[swap].contiguous())), torch.view_as_real(first[swap]))


@pytest.mark.parametrize("first", ["captured", "before"])
@pytest.mark.parametrize("shape,w", [((16, 16, 16), 6), ((8, 8, 8), 6), ((4, 4, 4), 10)])
def test_3d_captured_buffers_stay(afc, cuda, shape, w, first):
    # Both types captured, on a plan that has never run (per-point kernels: a
    # capture allocates nothing) or has run with as many points (its buffers'
    # addresses are in the graph); then larger calls, which grow the buffers
    # twice, and others' allocations in between.
    from apollofft_b200.nufft import NufftPlan3D
    npts = 1500
    g = torch.Generator(device="cuda").manual_seed(w)
    dims = torch.tensor(shape, dtype=torch.float64, device="cuda")
    pos = [(torch.rand(k * npts, 3, dtype=torch.float64, device="cuda", generator=g) * dims).contiguous()
           for k in (1, 3, 20)]
    val = [torch.randn(k * npts, dtype=torch.complex128, device="cuda", generator=g) for k in (1, 3, 20)]
    modes = torch.randn(shape, dtype=torch.complex128, device="cuda", generator=g)
    plan, other = (NufftPlan3D(shape, (1.0, 1.0, 1.0), 2, w) for _ in range(2))
    big = NufftPlan3D((4, 4, 4), (1.0, 1.0, 1.0), 2, 10)  # loads the per-point kernels outside a capture
    big.type2(big.type1(pos[0], val[0]), pos[0])
    want1, want2 = other.type1(pos[0], val[0]), other.type2(modes, pos[0])
    if first == "before":
        plan.type2(plan.type1(pos[0], val[0]), pos[0])
    out1, out2 = torch.zeros_like(want1), torch.zeros_like(want2)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.type1(pos[0], val[0], out=out1)
        plan.type2(modes, pos[0], out=out2)
    for k in (1, 2):
        got1, got2 = plan.type1(pos[k], val[k]), plan.type2(modes, pos[k])
        other.type1(pos[k], val[k])
        out1.zero_()
        out2.zero_()
        graph.replay()
        torch.cuda.synchronize()
        # sums of the same products in another order
        assert rel_l2(out1.cpu().numpy(), want1.cpu().numpy()) < 1e-13
        assert rel_l2(out2.cpu().numpy(), want2.cpu().numpy()) < 1e-13
        assert rel_l2(plan.type1(pos[k], val[k]).cpu().numpy(), got1.cpu().numpy()) < 1e-13
        assert torch.equal(torch.view_as_real(plan.type2(modes, pos[k])), torch.view_as_real(got2))
