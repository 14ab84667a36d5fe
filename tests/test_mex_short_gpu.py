"""Both gradients of short patches under many instances from one read of y and dy: edges of the 64 x 64 tiles and of the 8, 16 and
32 tap widths, vector and scalar staging, blocks that leave the input, gaps, and sums long enough for the fixed split."""
import importlib

import pytest
import torch

import cases
import gpu_util
from simnets_tf_b200 import abi

mex_ops = importlib.import_module("simnets_tf_b200.ops.mex")
pytestmark = pytest.mark.gpu

SHARED = dict(unshared=False, shared_region=(-1,))
EDGES = [
    cases.mex_case("taps_8_rows_64", (2, 4, 16, 16), 64, (2, 2, 2), (2, 2, 2), softmax=True, eps=0.5, seed=601, **SHARED),
    cases.mex_case("taps_9_rows_65", (3, 2, 12, 12), 65, (1, 3, 3), (1, 3, 3), softmax=True, seed=602, normalize=True, **SHARED),
    cases.mex_case("taps_16_rows_128", (2, 8, 10, 10), 128, (4, 2, 2), (4, 2, 2), eps=-0.7, seed=603, **SHARED),
    cases.mex_case("taps_17_odd", (3, 17, 5, 7), 50, (17, 1, 1), (17, 1, 1), softmax=True, seed=604, normalize=True, **SHARED),
    cases.mex_case("taps_32_rows_63", (1, 8, 8, 8), 63, (8, 2, 2), (8, 2, 2), softmax=True, eps=1.5, seed=605, **SHARED),
    cases.mex_case("regions", (2, 6, 12, 10), 70, (3, 2, 2), (3, 2, 2), softmax=True, unshared_region=(3,), seed=606, normalize=True),
    cases.mex_case("outside", (2, 6, 9, 11), 48, (2, 3, 2), (3, 3, 3), (1, 1, 1), oob=0.4, softmax=True, seed=607, **SHARED),
]


@pytest.mark.parametrize("c", EDGES, ids=lambda c: c["name"])
def test_tile_edges(port, c):
    gpu_util.check_mex(port, c, flags=abi.FLAG_MEX_NO_SMALL_TILES, f64_tiebreak=True)


def test_long_sums_agree_with_the_one_tile_kernels():
    """Beyond 1500 positions per accumulator the split is the one-tile kernel's, and so are the sums."""
    x = torch.randn(48, 2, 256, 256, device="cuda")
    attrs = dict(blocks=[1, 2, 4], strides=[1, 2, 4], epsilon=0.5, softmax_mode=True, use_unshared_regions=False, shared_offset_region=[-1])
    off = torch.randn(1, 64, 1, 2, 4, device="cuda")
    y = mex_ops.mex_forward(x, off, 64, **attrs)
    dy = torch.randn_like(y)
    dx, doff = mex_ops.mex_backward(x, off, y, dy, 64, **attrs)
    one_dx, one_doff = mex_ops.mex_backward(x, off, y, dy, 64, flags=abi.FLAG_MEX_TC_ONE_TILE, **attrs)
    assert float((doff - one_doff).norm()) <= 1e-5 * float(one_doff.norm())
    assert float((dx - one_dx).norm()) <= 1e-5 * float(one_dx.norm())


def test_long_sums_against_float64():
    """The tensor cores truncate what they add to an accumulator: each of its additions loses up to 2^-23 of it, and there are three
    (hi lo, lo hi, hi hi) for every eight positions of a share.  Shares are at least as many as multiprocessors."""
    x = torch.randn(48, 2, 256, 256, device="cuda")
    attrs = dict(blocks=[1, 2, 4], strides=[1, 2, 4], epsilon=0.5, softmax_mode=True, use_unshared_regions=False, shared_offset_region=[-1])
    off = torch.randn(1, 64, 1, 2, 4, device="cuda")
    y = mex_ops.mex_forward(x, off, 64, **attrs)
    dy = torch.randn_like(y)
    doff = mex_ops.mex_offsets_grad(x, off, y, dy, 64, **attrs)
    eo, want, positions = torch.exp(0.5 * off.double()).reshape(64, 8), 0, 0
    for n in range(48):                                     # disjoint blocks: sum over positions of dy * softmax weights
        patches = x[n].double().reshape(2, 128, 2, 64, 4).permute(0, 1, 3, 2, 4).reshape(-1, 8)
        ex = torch.exp(0.5 * (patches - patches.amax(1, keepdim=True)))
        q = dy[n].double().reshape(64, -1).t() / (ex @ eo.t())
        want = want + eo * (q.t() @ ex)
        positions += patches.shape[0]
    share = positions / torch.cuda.get_device_properties(0).multi_processor_count
    bound = 3 * (share / 8) * 2.0 ** -23 + 1e-6
    err = float((doff.reshape(64, 8).double() - want).norm() / want.norm())
    print("offsets gradient over %d positions: %.2e of its norm from float64 (bound %.2e)" % (positions, err, bound))
    assert err <= bound


@pytest.mark.parametrize("m,block", [(64, (2, 2, 2)), (100, (4, 2, 2)), (256, (8, 2, 2))], ids=["taps_8", "taps_16", "taps_32"])
def test_products_of_64_are_added_in_fp32(m, block):
    """Up to 1500 positions per accumulator of the one-tile kernels: what 64 positions (offsets gradient) or 64 instances (input
    gradient) contribute is added in FP32, so that neither gradient is farther from float64 than FP32 sums are (1e-6 of its norm; truncated
    additions would be at 3 / 8 x 2^-23 per position, 4e-5 at a thousand)."""
    attrs = dict(blocks=list(block), strides=list(block), epsilon=0.5, softmax_mode=True, use_unshared_regions=False, shared_offset_region=[-1])
    gen = torch.Generator(device="cuda").manual_seed(m)
    x, off = torch.randn(64, 16, 32, 32, generator=gen, device="cuda"), torch.randn((1, m) + block, generator=gen, device="cuda")
    y = mex_ops.mex_forward(x, off, m, flags=abi.FLAG_MEX_NO_SMALL_TILES, **attrs)
    dy = torch.randn(y.shape, generator=gen, device="cuda")
    got = mex_ops.mex_backward(x, off, y, dy, m, flags=abi.FLAG_MEX_NO_SMALL_TILES, **attrs)
    y64 = mex_ops.mex_forward(x.double(), off.double(), m, **attrs)
    want = mex_ops.mex_backward(x.double(), off.double(), y64, dy.double(), m, **attrs)
    for g, w in zip(got, want):
        assert float((g.double() - w).norm() / w.norm()) <= 1e-6
