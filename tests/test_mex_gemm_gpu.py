"""The small-contraction MEX kernels (float64 layers, small float32 layers, input gradients of overlapping blocks) at the
edges of their tiles, and the tensor-core kernels at the small sizes that would otherwise run on them."""
import ctypes as C
import importlib

import numpy as np
import pytest
import torch

import cases
import gpu_util
from simnets_tf_b200 import abi

mex_ops = importlib.import_module("simnets_tf_b200.ops.mex")
pytestmark = pytest.mark.gpu

# row counts around the tile heights 16, 32 and 64, tap counts around the 16-step chunks and the 64 columns, position counts
# around 64, reductions long enough to be split, overlapping and padded blocks, gaps between blocks
EDGES = [
    cases.mex_case("one_of_each", (1, 1, 1, 1), 1, (1, 1, 1), softmax=True, seed=501),
    cases.mex_case("rows_15_taps_17", (3, 17, 5, 5), 15, (17, 1, 1), (17, 1, 1), softmax=True, seed=502, normalize=True),
    cases.mex_case("rows_33_taps_65", (2, 65, 8, 9), 33, (65, 1, 1), (65, 1, 1), eps=0.5, softmax=True, unshared_region=(2,), seed=503, normalize=True),
    cases.mex_case("rows_65_split", (2, 130, 2, 2), 65, (130, 1, 1), (130, 1, 1), eps=-0.8, unshared_region=(2,), seed=504),
    cases.mex_case("positions_63", (1, 9, 9, 7), 20, (9, 1, 1), (9, 1, 1), softmax=True, unshared=False, shared_region=(-1,), seed=505),
    cases.mex_case("long_row", (2, 80, 4, 4), 3, (80, 4, 4), (80, 4, 4), softmax=True, seed=506, normalize=True),
    cases.mex_case("overlap_padded", (3, 5, 7, 8), 9, (3, 3, 2), (2, 1, 1), (1, 1, 1), oob=0.4, softmax=True, unshared_region=(2,), seed=507, normalize=True),
    cases.mex_case("overlap_strided", (2, 4, 11, 10), 18, (4, 5, 3), (4, 2, 2), (0, 2, 1), eps=1.5, unshared=False, shared_region=(2,), seed=508),
    cases.mex_case("gaps", (2, 6, 9, 9), 5, (2, 2, 2), (3, 3, 4), softmax=True, seed=509),
    # maps of a few pixels (lanes along instances), reductions split over clusters of two to eight CTAs and over more than a cluster holds
    cases.mex_case("map_2x2_split", (5, 150, 2, 2), 70, (150, 1, 1), (150, 1, 1), softmax=True, unshared_region=(2,), seed=510, normalize=True),
    cases.mex_case("map_2x2_many", (70, 33, 2, 2), 33, (33, 1, 1), (33, 1, 1), softmax=True, unshared_region=(2,), seed=511),
    cases.mex_case("map_1x1_cluster_of_8", (3, 500, 1, 1), 20, (500, 1, 1), (500, 1, 1), softmax=True, seed=512, normalize=True),
    cases.mex_case("map_1x1_11_splits", (3, 700, 1, 1), 129, (700, 1, 1), (700, 1, 1), eps=0.7, softmax=True, seed=513),
    cases.mex_case("map_3x3", (4, 40, 3, 3), 33, (40, 1, 1), (40, 1, 1), softmax=True, unshared=False, shared_region=(-1,), seed=514),
    cases.mex_case("whole_planes", (2, 90, 4, 4), 20, (90, 4, 4), (90, 4, 4), softmax=True, seed=515, normalize=True),
    # windows that overlap: also along channels, off the input on every side, in maps wider than the prepass holds and just not so
    cases.mex_case("overlap_channels", (2, 6, 9, 8), 11, (3, 2, 3), (2, 1, 2), (1, 1, 1), oob=0.7, eps=-1.2, unshared=False, shared_region=(2,), seed=516),
    cases.mex_case("overlap_wide_1", (1, 2, 5, 600), 3, (2, 3, 3), (2, 1, 1), (0, 1, 1), oob=-5.0, softmax=True, seed=517),
    cases.mex_case("overlap_wide_2", (1, 2, 4, 900), 3, (2, 3, 3), (2, 1, 1), (0, 1, 1), oob=5.0, softmax=True, seed=518),
    cases.mex_case("overlap_72_rows", (2, 8, 9, 9), 6, (8, 3, 3), (8, 1, 1), (0, 1, 1), softmax=True, unshared_region=(2,), seed=519),
]


@pytest.mark.parametrize("dtype", [abi.F32, abi.F64], ids=["f32", "f64"])
@pytest.mark.parametrize("c", EDGES, ids=lambda c: c["name"])
def test_tile_edges(port, c, dtype):
    gpu_util.check_mex(port, c, dtype=dtype, tol=1e-5 if dtype == abi.F32 else 1e-12, f64_tiebreak=dtype == abi.F32)


@pytest.mark.parametrize("c", cases.MEX_PAIR + cases.MEX_CONFIGS + cases.MEX_HEAD + cases.MEX_ROWS + [c for c in cases.MEX_SMALL if c["name"].startswith(("tc_", "tiled_", "head_"))],
                         ids=lambda c: c["name"])
def test_large_layer_kernels_at_small_sizes(port, c):
    gpu_util.check_mex(port, c, flags=abi.FLAG_MEX_NO_SMALL_TILES, f64_tiebreak=True)
    gpu_util.check_mex_pooled_dy(port, c, flags=abi.FLAG_MEX_NO_SMALL_TILES, tol=2e-5)


@pytest.mark.parametrize("flags", [0, abi.FLAG_MEX_NO_SMALL_TILES], ids=["small", "large"])
def test_overlapping_input_gradient_in_parts(flags):
    """More products than the workspace holds at a time: the batch is walked in parts, with the results of single samples."""
    x, off = torch.randn(12, 16, 128, 128, device="cuda"), torch.randn(1, 4, 16, 5, 5, device="cuda")
    attrs = dict(blocks=[16, 5, 5], strides=[16, 1, 1], padding=[0, 2, 2], softmax_mode=True, use_unshared_regions=False, shared_offset_region=[-1])
    y = mex_ops.mex_forward(x, off, 4, flags=flags, **attrs)
    dy = torch.randn_like(y)
    dx = mex_ops.mex_input_grad(x, off, y, dy, 4, flags=flags, **attrs)
    for n in (0, 9, 10, 11):
        one = mex_ops.mex_input_grad(x[n:n + 1], off, y[n:n + 1], dy[n:n + 1], 4, flags=flags, **attrs)
        assert torch.allclose(dx[n:n + 1], one, rtol=1e-5, atol=1e-5 * float(one.abs().max()))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64], ids=["f32", "f64"])
def test_products_of_overlapping_blocks_live_for_one_call(dtype):
    """Neither a forward call nor the workspace that a differentiated layer keeps has room for the products (189 or 252 MB here)."""
    x, off = torch.randn(12, 16, 128, 128, device="cuda", dtype=dtype), torch.randn(1, 4, 16, 3, 5, device="cuda", dtype=dtype, requires_grad=True)
    attrs = dict(blocks=[16, 3, 5], strides=[16, 1, 1], padding=[0, 1, 2], softmax_mode=True, use_unshared_regions=False, shared_offset_region=[-1])
    out = 4 * 12 * 128 * 128 * x.element_size()
    torch.cuda.synchronize()
    for x in (x, x.requires_grad_()):
        before = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        y = mex_ops.mex(x, off, 4, **attrs)
        assert torch.cuda.max_memory_allocated() - before < out + (16 << 20)
    torch.autograd.grad(y.sum(), (x, off))
    assert torch.cuda.max_memory_allocated() - before > 170 << 20


@pytest.mark.parametrize("dtype", [abi.F32, abi.F64], ids=["f32", "f64"])
@pytest.mark.parametrize("flags", [0, abi.FLAG_MEX_NO_SMALL_TILES], ids=["small", "large"])
@pytest.mark.parametrize("c", [c for c in EDGES if c["name"].startswith("overlap")], ids=lambda c: c["name"])
def test_scratch_of_exactly_the_stated_sizes(cuda_lib, c, flags, dtype):
    """Workspace and products fenced on both sides: nothing outside is written, and results do not depend on what was inside."""
    def fenced(n, fill):
        t = torch.full((n + 512,), fill, dtype=torch.uint8, device="cuda")
        t[:256], t[256 + n:] = 0x5A, 0x5A
        return t, t.data_ptr() + 256

    np_t, t_t = (np.float32, torch.float32) if dtype == abi.F32 else (np.float64, torch.float64)
    d = cases.mex_desc(c, dtype=dtype)
    d.flags |= flags
    g = abi.MexGeometry()
    assert cuda_lib.simnets_mex_dims(C.byref(d), C.byref(g)) == 0
    oshape = (c["shape"][0], g.channels_out_total, g.height_out, g.width_out)
    x, off, dy = (gpu_util.dev(a, t_t) for a in cases.mex_inputs(c, (g.num_regions, g.M, g.block_c, g.block_h, g.block_w), oshape, np_t))
    kept, products = cuda_lib.simnets_mex_forward_workspace_bytes(C.byref(d)), cuda_lib.simnets_mex_products_bytes(C.byref(d))
    assert products > 0
    stream, got = torch.cuda.current_stream().cuda_stream, []
    for fill in (0, 0xFF):
        (ws, wp), (pr, pp) = fenced(kept, fill), fenced(products, fill)
        y, dx, doff = torch.empty(oshape, dtype=t_t, device="cuda"), torch.empty_like(x), torch.empty_like(off)
        assert cuda_lib.simnets_mex_forward(C.byref(d), x.data_ptr(), off.data_ptr(), y.data_ptr(), wp, kept, stream) == 0
        args = [C.byref(d), x.data_ptr(), off.data_ptr(), y.data_ptr(), dy.data_ptr(), dx.data_ptr(), doff.data_ptr(), wp]
        assert cuda_lib.simnets_mex_gradients(*args, kept, pp, products - 256, stream) == abi.E_WORKSPACE
        assert cuda_lib.simnets_mex_gradients(*args, 256, pp, products, stream) == abi.E_WORKSPACE
        assert cuda_lib.simnets_mex_gradients(*args, kept, pp, products, stream) == 0
        for t, n in ((ws, kept), (pr, products)):
            assert bool((t[:256] == 0x5A).all()) and bool((t[256 + n:] == 0x5A).all())
        got.append((y, dx, doff))
        one = torch.empty(kept + products, dtype=torch.uint8, device="cuda")
        dx2, doff2 = torch.empty_like(dx), torch.empty_like(doff)
        args = [C.byref(d), x.data_ptr(), off.data_ptr(), y.data_ptr(), dy.data_ptr(), dx2.data_ptr(), doff2.data_ptr(), one.data_ptr()]
        assert cuda_lib.simnets_mex_backward(*args, kept + products, stream) == 0
        got.append((y, dx2, doff2))
    for other in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0], other))


@pytest.mark.parametrize("shape,m", [((3, 12, 6, 6), 10), ((3, 200, 2, 2), 20), ((2, 700, 1, 1), 18)], ids=["one", "cluster", "splits"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64], ids=["f32", "f64"])
def test_offsets_beyond_the_safe_spread_are_evaluated_term_by_term(port, dtype, shape, m):
    c = cases.mex_case("spread", shape, m, (shape[1], 1, 1), (shape[1], 1, 1), softmax=True, unshared_region=(2 if shape[2] > 1 else 1,), seed=520)
    code = abi.F32 if dtype == torch.float32 else abi.F64
    d = cases.mex_desc(c, dtype=code)
    x, off, dy = cases.mex_inputs(c, port.mex_offsets_shape(d), port.mex_out_shape(d), np.float32 if code == abi.F32 else np.float64)
    off[off.shape[0] // 2, 3, 5] = -500.0
    xd, od, dyd = (gpu_util.dev(a, dtype) for a in (x, off, dy))
    attrs = cases.mex_attrs(c)
    ry = port.mex_forward(d, x, off)
    cases.assert_parity(mex_ops.mex_forward(xd, od, c["M"], **attrs).cpu().numpy(), ry, what="y")
    dx, doff = mex_ops.mex_backward(xd, od, gpu_util.dev(ry, dtype), dyd, c["M"], **attrs)
    cases.assert_parity(dx.cpu().numpy(), port.mex_input_grad(d, x, off, ry, dy), what="dx")
    cases.assert_parity(doff.cpu().numpy(), port.mex_offsets_grad(d, x, off, ry, dy), tol=2e-5, what="doff")


# just above the line of the small layers, too few instances for the tensor cores: the forward pass of other kernels, the gradients of these
BACKWARD_ONLY = [
    cases.mex_case("short_patches", (24, 32, 32, 32), 8, (4, 2, 2), (4, 2, 2), softmax=True, unshared=False, shared_region=(-1,), seed=530),
    cases.mex_case("pixels", (40, 33, 20, 22), 47, (33, 1, 1), (33, 1, 1), softmax=True, unshared_region=(2,), seed=531, normalize=True),
    cases.mex_case("gaps_padded", (16, 20, 30, 32), 30, (10, 3, 2), (10, 4, 2), (0, 2, 1), oob=0.3, eps=0.6, unshared_region=(2,), seed=532),
]


@pytest.mark.parametrize("c", BACKWARD_ONLY, ids=lambda c: c["name"])
def test_gradients_behind_another_family_s_forward_pass(port, c):
    """float64 of the same kernels as the reference; calls that share one primed workspace, in either order, give the same."""
    d = cases.mex_desc(c)
    x, off, dy = (gpu_util.dev(a) for a in cases.mex_inputs(c, port.mex_offsets_shape(d), port.mex_out_shape(d)))
    attrs, m = cases.mex_attrs(c), c["M"]
    ws = mex_ops.mex_layer_workspace(x, m, flags=0, **attrs)
    ws.fill_(0xFF)
    y = mex_ops.mex_forward(x, off, m, workspace=ws, **attrs)
    wide = mex_ops.mex_forward(x.double(), off.double(), m, **attrs)
    assert float((y.double() - wide).abs().max()) <= 1e-5 * float(wide.abs().max())
    want = mex_ops.mex_backward(x.double(), off.double(), wide, dy.double(), m, **attrs)
    doff = mex_ops.mex_offsets_grad(x, off, y, dy, m, primed_workspace=ws, **attrs)
    dx = mex_ops.mex_input_grad(x, off, y, dy, m, primed_workspace=ws, **attrs)
    both = mex_ops.mex_backward(x, off, y, dy, m, primed_workspace=ws, **attrs)
    alone = mex_ops.mex_backward(x, off, y, dy, m, **attrs)
    for got, other, third, ref in zip((dx, doff), both, alone, want):
        assert torch.equal(got, other) and torch.equal(got, third)
        assert float((got.double() - ref).norm()) <= 2e-6 * float(ref.norm())
    old = mex_ops.mex_backward(x, off, y, dy, m, flags=abi.FLAG_MEX_NO_SMALL_TILES, **attrs)
    for got, other in zip((dx, doff), old):
        assert float((got - other).norm()) <= 2e-5 * float(other.norm())
    if y.shape[2] % 2 == 0 and y.shape[3] % 2 == 0:
        small = torch.randn(y.shape[0], y.shape[1], y.shape[2] // 2, y.shape[3] // 2, device="cuda")
        full = small.repeat_interleave(2, 2).repeat_interleave(2, 3).contiguous()
        for a, b in zip(mex_ops.mex_backward(x, off, y, small, m, pooled=True, **attrs), mex_ops.mex_backward(x, off, y, full, m, **attrs)):
            assert torch.equal(a, b)


@pytest.mark.parametrize("shape,m,blocks,regions", [((28, 64, 32, 32), 8, (4, 2, 2), 0), ((48, 32, 32, 32), 30, (32, 1, 1), 2), ((40, 12, 24, 25), 9, (12, 3, 3), 0)],
                         ids=["short_patches", "pixels", "overlapping"])
def test_long_sums_beyond_the_safe_spread(shape, m, blocks, regions):
    """One offset 200 below the others, up to 115 K positions in a sum of the offsets gradient.  256 threads share them: a register of up to 450
    terms is some 0.3 x 2^-24 x sqrt(450) = 4e-7 of its sum away from it, one that takes all terms 6e-6."""
    strides = blocks if blocks[1] < 3 else (blocks[0], 1, 1)
    region = dict(use_unshared_regions=True, unshared_offset_region=[regions]) if regions else dict(use_unshared_regions=False, shared_offset_region=[-1])
    attrs = dict(softmax_mode=True, blocks=list(blocks), strides=list(strides), **region)
    gen = torch.Generator(device="cuda").manual_seed(m)
    x, off = torch.randn(shape, generator=gen, device="cuda"), torch.randn((max(1, regions) ** 2, m) + blocks, generator=gen, device="cuda")
    off[-1, m // 2, 1, 0, 0] = -200.0
    y = mex_ops.mex_forward(x.double(), off.double(), m, flags=abi.FLAG_FORCE_DIRECT, **attrs)
    dy = torch.randn(y.shape, generator=gen, device="cuda")
    want = mex_ops.mex_backward(x.double(), off.double(), y, dy.double(), m, flags=abi.FLAG_FORCE_DIRECT, **attrs)
    wide = mex_ops.mex_backward(x.double(), off.double(), y, dy.double(), m, **attrs)
    for got, ref in zip(wide, want):
        assert float((got - ref).norm()) <= 1e-14 * float(ref.norm())
    y = y.float()
    want = mex_ops.mex_backward(x.double(), off.double(), y.double(), dy.double(), m, flags=abi.FLAG_FORCE_DIRECT, **attrs)
    for got, ref in zip(mex_ops.mex_backward(x, off, y, dy, m, **attrs), want):
        assert float((got.double() - ref).norm()) <= 1.5e-6 * float(ref.norm())


@pytest.mark.parametrize("dtype", [abi.F32, abi.F64], ids=["f32", "f64"])
@pytest.mark.parametrize("c", BACKWARD_ONLY + [c for c in EDGES if c["name"] in ("overlap_72_rows", "map_2x2_split")], ids=lambda c: c["name"])
def test_status_words_of_gradients_on_a_fresh_workspace(cuda_lib, c, dtype):
    """A gradient call without a forward pass in front runs the prepass itself, and says what that found."""
    t_t = torch.float32 if dtype == abi.F32 else torch.float64
    d = cases.mex_desc(c, dtype=dtype)
    g = abi.MexGeometry()
    assert cuda_lib.simnets_mex_dims(C.byref(d), C.byref(g)) == 0
    oshape = (c["shape"][0], g.channels_out_total, g.height_out, g.width_out)
    x, off, dy = (gpu_util.dev(a, t_t) for a in cases.mex_inputs(c, (g.num_regions, g.M, g.block_c, g.block_h, g.block_w), oshape))
    bytes_, stream, status = cuda_lib.simnets_mex_workspace_bytes(C.byref(d)), torch.cuda.current_stream().cuda_stream, (C.c_int32 * 2)(7, 7)
    for spread, want in ((0.0, 0), (-700.0, 1)):
        off[0, 0, 0, 0, 0] += spread
        y = mex_ops.mex_forward(x, off, c["M"], **cases.mex_attrs(c))
        dx, doff = torch.empty_like(x), torch.empty_like(off)
        tensors = [C.byref(d), x.data_ptr(), off.data_ptr(), y.data_ptr(), dy.data_ptr()]
        for call, out in ((cuda_lib.simnets_mex_input_grad, [dx.data_ptr()]), (cuda_lib.simnets_mex_offsets_grad, [doff.data_ptr()]),
                          (cuda_lib.simnets_mex_backward, [dx.data_ptr(), doff.data_ptr()])):
            ws = torch.full((bytes_,), 0xFF, dtype=torch.uint8, device="cuda")
            assert call(*tensors, *out, ws.data_ptr(), bytes_, stream) == 0
            assert cuda_lib.simnets_mex_workspace_status(ws.data_ptr(), stream, status) == 0
            torch.cuda.synchronize()
            assert tuple(status) == (want, 0)
