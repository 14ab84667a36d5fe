"""The float32 Similarity kernels where they can go wrong: tap, template and channel counts around the tile sizes, strides whose
phases have different taps and pixels, pixels that no patch covers, inputs small and large enough for every dispatch."""
import numpy as np
import pytest
import torch

import cases
import gpu_util

pytestmark = pytest.mark.gpu

NAN = cases.NAN
MODES = [dict(fn="L2"), dict(fn="L2", norm=True), dict(fn="L2", norm=True, ignore_nan=True, nan_frac=0.2), dict(fn="L1")]
# (batch, channels, h, w), templates, blocks, strides, padding
SHAPES = [
    ((1, 1, 5, 6), 1, (1, 1), (1, 1), (0, 0)),              # one tap
    ((2, 5, 7, 9), 33, (1, 1), (1, 1), (0, 0)),             # five taps, up to eight channels
    ((2, 3, 11, 10), 65, (3, 3), (1, 1), (1, 1)),           # 27 taps
    ((1, 8, 9, 8), 31, (2, 2), (1, 1), (1, 1)),             # 32 taps, 8 channels
    ((2, 9, 10, 7), 64, (2, 2), (2, 2), (1, 1)),            # 36 taps, 9 channels, four phases
    ((1, 16, 8, 9), 32, (2, 2), (1, 2), (0, 1)),            # 64 taps
    ((2, 13, 9, 11), 40, (5, 1), (2, 1), (2, 0)),           # 65 taps, uneven phases
    ((1, 17, 12, 9), 20, (3, 2), (4, 3), (0, 0)),           # gaps: pixels that no patch covers
    ((2, 33, 6, 7), 50, (2, 2), (1, 1), (1, 1)),            # 132 taps, 33 channels
    ((1, 66, 5, 6), 129, (1, 2), (1, 1), (0, 1)),           # 66 channels, 129 templates
    ((1, 130, 4, 5), 12, (1, 1), (1, 1), (0, 0)),           # 130 channels
]


@pytest.mark.parametrize("mode", MODES, ids=["l2", "l2n", "l2nan", "l1"])
@pytest.mark.parametrize("i", range(len(SHAPES)))
def test_tile_edges(port, i, mode):
    shape, M, blocks, strides, padding = SHAPES[i]
    gpu_util.check_similarity(port, cases.sim_case("edges%d" % i, shape, M, blocks=blocks, strides=strides, padding=padding, oob=0.3, seed=700 + i, **mode),
                              f64_tiebreak=True)


@pytest.mark.parametrize("mode", MODES, ids=["l2", "l2n", "l2nan", "l1"])
@pytest.mark.parametrize("shape,M,blocks", [((160, 1, 28, 28), 40, (2, 2)), ((96, 3, 30, 33), 10, (3, 3))], ids=["resident_32", "many_pixels"])
def test_enough_positions_for_the_streaming_kernels(port, shape, M, blocks, mode):
    gpu_util.check_similarity(port, cases.sim_case("many", shape, M, blocks=blocks, strides=(1, 1), padding=(1, 1), seed=720, **mode), f64_tiebreak=True, tol=2e-5)


@pytest.mark.parametrize("mode", MODES, ids=["l2", "l2n", "l2nan", "l1"])
@pytest.mark.parametrize("i", range(len(SHAPES)))
def test_infinite_pixels_meet_only_the_taps_that_are_there(port, i, mode):
    """With dy >= 0 an infinite pixel has an infinite gradient; a tap cut off by the padding, or a step past the last one, must
    not turn it into NaN."""
    shape, M, blocks, strides, padding = SHAPES[i]
    c = cases.sim_case("inf%d" % i, shape, M, blocks=blocks, strides=strides, padding=padding, oob=0.3, seed=740 + i, **mode)
    d = cases.sim_desc(c)
    x, t, w, dy = cases.sim_inputs(c, port.sim_out_shape(d))
    rng = np.random.default_rng(i)
    x[rng.random(x.shape) < 0.2] = np.inf
    x[rng.random(x.shape) < 0.1] = -np.inf
    dy = np.abs(dy)
    dx = gpu_util.sim_ops.similarity_input_grad(*(gpu_util.dev(a) for a in (x, t, w, dy)), **cases.sim_attrs(c)).cpu().numpy()
    ref = port.similarity_input_grad(d, x, t, w, dy)
    assert np.isinf(ref).any() or mode["fn"] == "L1"
    cases.assert_parity(dx, ref, what=c["name"])


# rows of channels per tile: 16, 20, 24, 32, 40, 48, 64; instances per chunk: 8, and 16 for 64 rows, four steps at a time
@pytest.mark.parametrize("mode", MODES, ids=["l2", "l2n", "l2nan", "l1"])
@pytest.mark.parametrize("channels,m", [(16, 9), (17, 1), (20, 8), (21, 4), (24, 5), (25, 12), (32, 7), (33, 17), (40, 16), (41, 3), (48, 10), (49, 15), (64, 16), (65, 20),
                                        (63, 33), (80, 4), (97, 13), (128, 31), (129, 5)])
def test_input_gradients_at_the_edges_of_their_tiles(port, channels, m, mode):
    c = cases.sim_case("rows%d" % channels, (2, channels, 9, 8), m, blocks=(3, 2), strides=(2, 1), padding=(1, 0), oob=0.3, seed=800 + channels, **mode)
    d = cases.sim_desc(c)
    x, t, w, dy = cases.sim_inputs(c, port.sim_out_shape(d))
    x[0, :, 2, 3] = t[0, :, 1, 1]                          # (differences of exactly 0)
    dx = gpu_util.sim_ops.similarity_input_grad(*(gpu_util.dev(a) for a in (x, t, w, dy)), **cases.sim_attrs(c)).cpu().numpy()
    a64 = [a.astype(np.float64) for a in (x, t, w, dy)]
    cases.assert_parity(dx, port.similarity_input_grad(d, x, t, w, dy), port.similarity_input_grad(cases.sim_desc(c, dtype=gpu_util.abi.F64), *a64), what=c["name"])


# One FP32 register is about 0.3 x 2^-24 x sqrt(n) of a sum of n such terms away from it (measured: n = 252: 2.8e-7, n = 6400: 1.4e-6).
def _of_folded(steps, folds):
    return 0.3 * 2.0 ** -24 * (steps ** 0.5 + folds ** 0.5)


@pytest.mark.parametrize("attrs", [dict(), dict(normalization_term=True), dict(normalization_term=True, ignore_nan_input=True), dict(similarity_function="L1")],
                         ids=["l2", "l2n", "l2nan", "l1"])
@pytest.mark.parametrize("channels,strides,m", [(3, 1, 256), (12, 1, 256), (40, 1, 256), (40, 4, 256), (40, 1, 11), (70, 1, 256), (130, 1, 100)],
                         ids=["narrow", "rows16", "rows64", "gaps", "one_aside", "rows128", "two_chunks"])
def test_input_gradients_of_long_sums_are_folded(channels, strides, m, attrs):
    """Up to 25 x 256 steps, set aside every 256 of them."""
    gen = torch.Generator(device="cuda").manual_seed(m)
    x, t = torch.randn(2, channels, 20, 20, generator=gen, device="cuda"), 0.1 * torch.randn(m, channels, 5, 5, generator=gen, device="cuda")
    w = 1 + 0.1 * torch.rand(t.shape, generator=gen, device="cuda")
    kw = dict(blocks=[5, 5], strides=[strides, strides], padding=[0, 0], **attrs)
    out = 15 // strides + 1
    dy = torch.randn(2, m, out, out, generator=gen, device="cuda")
    want = gpu_util.sim_ops.similarity_input_grad(x.double(), t.double(), w.double(), dy.double(), **kw)
    got = gpu_util.sim_ops.similarity_input_grad(x, t, w, dy, **kw).double()
    assert float((got - want).norm() / want.norm()) <= _of_folded(256, 25)


@pytest.mark.parametrize("attrs", [dict(), dict(normalization_term=True), dict(normalization_term=True, ignore_nan_input=True), dict(similarity_function="L1")],
                         ids=["l2", "l2n", "l2nan", "l1"])
@pytest.mark.parametrize("m,channels,block,batch", [(256, 32, 3, 128), (64, 3, 3, 2048), (32, 1, 2, 8192), (64, 64, 3, 72), (64, 64, 3, 74)],
                         ids=["wide", "image", "copies", "few_aside", "one_more"])
def test_parameter_gradients_of_long_sums_are_folded(m, channels, block, batch, attrs):
    """Up to 60000 positions of a split, set aside every 2048 of them."""
    gen = torch.Generator(device="cuda").manual_seed(batch)
    x, t = torch.randn(batch, channels, 32, 32, generator=gen, device="cuda"), 0.1 * torch.randn(m, channels, block, block, generator=gen, device="cuda")
    w = 1 + 0.1 * torch.rand(t.shape, generator=gen, device="cuda")
    kw = dict(blocks=[block, block], strides=[1, 1], padding=[0, 0], **attrs)
    dy = torch.randn(batch, m, 33 - block, 33 - block, generator=gen, device="cuda")
    want = [0, 0]
    for i in range(0, batch, 512):
        for k, g in enumerate(gpu_util.sim_ops.similarity_parameters_grad(x[i:i + 512].double(), t.double(), w.double(), dy[i:i + 512].double(), **kw)):
            want[k] = want[k] + g
    for g, e in zip(gpu_util.sim_ops.similarity_parameters_grad(x, t, w, dy, **kw), want):
        assert float((g.double() - e).norm() / e.norm()) <= _of_folded(2048, 32)


# parameter gradients on 64 templates x 32 or 64 taps: (batch, channels, h, w), templates, blocks, strides, padding
PARAM_TILES = [
    ((1, 17, 6, 5), 33, (1, 1), (1, 1), (0, 0)),            # 17 taps, one chunk
    ((2, 8, 9, 7), 64, (2, 2), (1, 1), (1, 1)),             # 32 taps
    ((2, 11, 8, 9), 65, (3, 1), (1, 2), (1, 0)),            # 33 taps, a second row tile of one template
    ((3, 16, 7, 8), 100, (2, 2), (2, 1), (0, 1)),           # 64 taps
    ((2, 13, 9, 6), 70, (1, 5), (1, 1), (0, 2)),            # 65 taps: three tiles of 22
    ((2, 43, 5, 6), 130, (3, 1), (1, 1), (1, 0)),           # 129 taps: five tiles of 26
    ((2, 2, 17, 12), 40, (16, 1), (1, 1), (8, 0)),          # blocks of sixteen rows
    ((2, 2, 18, 9), 40, (17, 1), (1, 1), (8, 0)),           # and of seventeen, which take the smaller tiles
    ((40, 3, 13, 11), 64, (3, 3), (1, 1), (1, 1)),          # several chunks set aside
]


@pytest.mark.parametrize("mode", MODES, ids=["l2", "l2n", "l2nan", "l1"])
@pytest.mark.parametrize("special", [False, True], ids=["plain", "special"])
@pytest.mark.parametrize("i", range(len(PARAM_TILES)))
def test_parameter_gradients_at_the_edges_of_their_tiles(port, i, special, mode):
    """special: values that equal a template's (the sign of a difference of 0 is 0), with L1 also infinities and NaN."""
    shape, M, blocks, strides, padding = PARAM_TILES[i]
    c = cases.sim_case("params%d" % i, shape, M, blocks=blocks, strides=strides, padding=padding, oob=0.0 if special else 0.3, seed=760 + i, **mode)
    d = cases.sim_desc(c)
    x, t, w, dy = cases.sim_inputs(c, port.sim_out_shape(d))
    if special:
        rng = np.random.default_rng(i)
        x = np.where(rng.random(x.shape) < 0.1, rng.choice(t.reshape(-1), x.shape), x).astype(np.float32)
        if mode["fn"] == "L1":
            x[0, 0, 0, 0], x[0, 0, 1, 1], x[0, 0, 2, 2], t[1, 0, 0, 0] = np.inf, NAN, -np.inf, np.inf
    got = gpu_util.sim_ops.similarity_parameters_grad(*(gpu_util.dev(a) for a in (x, t, w, dy)), **cases.sim_attrs(c))
    d64 = cases.sim_desc(c, dtype=gpu_util.abi.F64)
    for g, ref, ref64 in zip(got, port.similarity_params_grad(d, x, t, w, dy), port.similarity_params_grad(d64, *(a.astype(np.float64) for a in (x, t, w, dy)))):
        cases.assert_parity(g.cpu().numpy(), ref, ref64, what=c["name"])


@pytest.mark.parametrize("mode", MODES, ids=["l2", "l2n", "l2nan", "l1"])
@pytest.mark.parametrize("blocks,padding,stride", [((16, 1), (15, 0), 1), ((1, 16), (0, 15), 2), ((17, 1), (16, 0), 1), ((1, 18), (0, 9), 1), ((16, 16), (8, 8), 3)],
                         ids=["rows16", "columns16", "rows17", "columns18", "square16"])
@pytest.mark.parametrize("batch,m", [(2, 7), (120, 33)], ids=["few", "many"])
def test_patches_that_leave_the_image_on_every_side(port, batch, m, blocks, padding, stride, mode):
    """Blocks up to and beyond sixteen rows or columns (how a tap is tested against the image changes there), patches almost entirely
    outside, on the kernels for few and for many positions."""
    size = (batch, 1, 21, 20) if blocks[0] * blocks[1] < 100 else (max(1, batch // 40), 1, 21, 20)
    c = cases.sim_case("leaves", size, m, blocks=blocks, strides=(stride, stride), padding=padding, oob=0.3, seed=850, **mode)
    d = cases.sim_desc(c)
    x, t, w, _ = cases.sim_inputs(c, port.sim_out_shape(d))
    y = gpu_util.sim_ops.similarity_forward(*(gpu_util.dev(a) for a in (x, t, w)), **cases.sim_attrs(c)).cpu().numpy()
    cases.assert_parity(y, port.similarity_forward(d, x, t, w), port.similarity_forward(cases.sim_desc(c, dtype=gpu_util.abi.F64), *(a.astype(np.float64) for a in (x, t, w))),
                        what=c["name"])


# ---- L1 where dy (or a weight) is no finite number and a difference is 0: 0 times it is NaN, on every kernel
L1_MODES = [dict(fn="L1"), dict(fn="L1", flags=gpu_util.abi.FLAG_SIM_L1_SKIP_NAN)]


def _l1_case(name, shape, M, blocks, strides, padding, seed, mode):
    c = cases.sim_case(name, shape, M, blocks=blocks, strides=strides, padding=padding, oob=0.3, seed=seed, **mode)
    return c, cases.sim_desc(c)


@pytest.mark.parametrize("mode", L1_MODES, ids=["l1", "l1skip"])
@pytest.mark.parametrize("channels", [5, 12, 17, 24, 30, 40, 48, 64, 70])
def test_l1_input_gradients_of_a_dy_that_is_no_number(port, channels, mode):
    """A patch of every sample is template 1, whose dy there is inf, NaN or -inf; one pixel equals a tap of infinite weight."""
    c, d = _l1_case("dy%d" % channels, (3, channels, 9, 8), 11, (3, 2), (2, 1), (1, 0), 870 + channels, mode)
    x, t, w, dy = cases.sim_inputs(c, port.sim_out_shape(d))
    for n, bad in enumerate((np.inf, NAN, -np.inf)):
        x[n, :, 3:6, 2:4] = t[1]                            # (output row 2, column 2)
        dy[n, 1, 2, 2] = bad
    x[0, :, 0, 6] = t[2, :, 1, 1]                           # (output row 0, column 5)
    w[2, 0, 1, 1] = np.inf
    dx = gpu_util.sim_ops.similarity_input_grad(*(gpu_util.dev(a) for a in (x, t, w, dy)), flags=c["flags"], **cases.sim_attrs(c)).cpu().numpy()
    ref = port.similarity_input_grad(d, x, t, w, dy)
    assert np.isnan(ref[:, :, 3:6, 2:4]).all() and np.isnan(ref[0, 0, 0, 6])
    cases.assert_parity(dx, ref, what=c["name"])


@pytest.mark.parametrize("mode", L1_MODES, ids=["l1", "l1skip"])
@pytest.mark.parametrize("channels,m", [(3, 33), (5, 64), (6, 40), (11, 70), (30, 100), (3, 20), (2, 40)])
def test_l1_parameter_gradients_of_a_dy_that_is_no_number(port, channels, m, mode):
    """The first channel of a patch of every sample is that of template 1, whose dy there is inf, NaN or -inf; 64 x 32 and 64 x 64 tiles, and
    the smaller ones of few templates or taps."""
    c, d = _l1_case("dp%d_%d" % (channels, m), (3, channels, 9, 8), m, (3, 2), (2, 1), (1, 0), 880 + channels, mode)
    x, t, w, dy = cases.sim_inputs(c, port.sim_out_shape(d))
    for n, bad in enumerate((np.inf, NAN, -np.inf)):
        x[n, 0, 3:6, 2:4] = t[1 + n, 0]                     # (output row 2, column 2)
        dy[n, 1 + n, 2, 2] = bad
    got = gpu_util.sim_ops.similarity_parameters_grad(*(gpu_util.dev(a) for a in (x, t, w, dy)), flags=c["flags"], **cases.sim_attrs(c))
    ref = port.similarity_params_grad(d, x, t, w, dy)
    assert np.isnan(ref[0][1:4, 0]).all() and np.isinf(ref[0][1, 1:]).all()
    for g, r in zip(got, ref):
        cases.assert_parity(g.cpu().numpy(), r, what=c["name"])


@pytest.mark.parametrize("i", range(len(PARAM_TILES)))
def test_l1_skipping_nan_at_the_edges_of_the_tiles(port, i):
    shape, M, blocks, strides, padding = PARAM_TILES[i]
    gpu_util.check_similarity(port, cases.sim_case("skip%d" % i, shape, M, blocks=blocks, strides=strides, padding=padding, oob=0.3, nan_frac=0.2, seed=890 + i, **L1_MODES[1]),
                              f64_tiebreak=True)


# ---- input gradients of a few templates: chunks of eight or sixteen steps that run through the taps, in tiles of 16, 32 and 64 rows
@pytest.mark.parametrize("infinite", [False, True], ids=["finite", "infinite"])
@pytest.mark.parametrize("mode", MODES + L1_MODES[1:], ids=["l2", "l2n", "l2nan", "l1", "l1skip"])
@pytest.mark.parametrize("channels,m,blocks,strides,padding", [
    (9, 1, (1, 1), (1, 1), (0, 0)), (12, 1, (3, 3), (1, 1), (1, 1)), (16, 3, (3, 2), (2, 1), (1, 0)), (24, 2, (5, 3), (1, 1), (2, 1)), (33, 1, (2, 2), (3, 3), (0, 0)),
    (32, 2, (3, 3), (2, 2), (1, 1)), (64, 1, (3, 3), (1, 1), (1, 1)), (64, 3, (5, 5), (1, 2), (2, 2)), (66, 5, (3, 3), (1, 1), (0, 1)), (128, 6, (3, 2), (2, 1), (1, 0)), (64, 7, (1, 1), (1, 1), (0, 0))])
def test_input_gradients_of_a_few_templates(port, channels, m, blocks, strides, padding, mode, infinite):
    c = cases.sim_case("few%d" % channels, (3, channels, 9, 8), m, blocks=blocks, strides=strides, padding=padding, oob=0.3, seed=900 + channels, **mode)
    d = cases.sim_desc(c)
    x, t, w, dy = cases.sim_inputs(c, port.sim_out_shape(d))
    if infinite:
        x[np.random.default_rng(m).random(x.shape) < 0.2] = np.inf
        dy = np.abs(dy)
    dx = gpu_util.sim_ops.similarity_input_grad(*(gpu_util.dev(a) for a in (x, t, w, dy)), flags=c["flags"], **cases.sim_attrs(c)).cpu().numpy()
    a64 = [a.astype(np.float64) for a in (x, t, w, dy)]
    cases.assert_parity(dx, port.similarity_input_grad(d, x, t, w, dy), port.similarity_input_grad(cases.sim_desc(c, dtype=gpu_util.abi.F64), *a64), what=c["name"])
