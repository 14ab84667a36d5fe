"""Samples whose values outnumber 32-bit offsets.  A stride picks few positions out of such a sample; the same positions gathered
into a small sample have the same patches, and a kernel that is the same for both gives the same values bit for bit."""
import pytest
import torch

import gpu_util

pytestmark = pytest.mark.gpu


def _parameters(m, c, bh, bw):
    gen = torch.Generator(device="cuda").manual_seed(m)
    t = torch.rand(m, c, bh, bw, generator=gen, device="cuda") - 0.5
    return t, 0.5 + torch.rand(m, c, bh, bw, generator=gen, device="cuda")


def _sample(*shape):
    return torch.rand(shape, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")


@pytest.mark.parametrize("attrs", [dict(), dict(normalization_term=True, ignore_nan_input=True), dict(similarity_function="L1")], ids=["l2", "l2nan", "l1"])
@pytest.mark.parametrize("m", [64, 20], ids=["rows64", "rows32"])
def test_offsets_of_channels_beyond_31_bits_of_bytes(m, attrs):
    """Three channels of 2^28 pixels: the third begins 2^31 bytes into the sample."""
    x, (t, w) = _sample(1, 3, 1 << 14, 1 << 14), _parameters(m, 3, 1, 1)
    y = gpu_util.sim_ops.similarity_forward(x, t, w, blocks=[1, 1], strides=[56, 56], padding=[0, 0], **attrs)
    few = x[:, :, ::56, ::56].contiguous()
    assert torch.equal(y, gpu_util.sim_ops.similarity_forward(few, t, w, blocks=[1, 1], strides=[1, 1], padding=[0, 0], **attrs))


def test_offsets_of_rows_beyond_31_bits_of_bytes():
    """Blocks of seventeen rows (tested against the image by ranges, not bits), 2^27 bytes apart."""
    x, (t, w) = _sample(1, 1, 17, 1 << 25), _parameters(64, 1, 17, 1)
    y = gpu_util.sim_ops.similarity_forward(x, t, w, blocks=[17, 1], strides=[1, 512], padding=[0, 0])
    few = x[:, :, :, ::512].contiguous()
    assert torch.equal(y, gpu_util.sim_ops.similarity_forward(few, t, w, blocks=[17, 1], strides=[1, 1], padding=[0, 0]))


@pytest.mark.parametrize("attrs", [dict(), dict(normalization_term=True, ignore_nan_input=True), dict(similarity_function="L1")], ids=["l2", "l2nan", "l1"])
def test_parameter_gradients_of_offsets_beyond_31_bits(attrs):
    """33 channels of 8200 x 8200 pixels: the last one begins 2^31 values into the sample.  Such samples go to the shape-agnostic kernel, which
    takes eight taps per block of the small one."""
    x, (t, w) = _sample(1, 33, 8200, 8200), _parameters(32, 33, 1, 1)
    few = x[:, :, ::64, ::64].contiguous()
    dy = torch.randn(1, 32, 129, 129, generator=torch.Generator(device="cuda").manual_seed(2), device="cuda")
    got = gpu_util.sim_ops.similarity_parameters_grad(x, t, w, dy, blocks=[1, 1], strides=[64, 64], padding=[0, 0], **attrs)
    want = gpu_util.sim_ops.similarity_parameters_grad(few, t, w, dy, blocks=[1, 1], strides=[1, 1], padding=[0, 0], flags=gpu_util.abi.FLAG_FORCE_DIRECT, **attrs)
    for a, b in zip(got, want):
        assert torch.equal(a, b)


def test_blocks_of_rows_beyond_a_wide_image():
    """Sixteen rows of 2^26 pixels around an image of two: most of the block lies outside, where its offsets need 32 bits and more."""
    x, dy = _sample(1, 1, 2, 1 << 26), None
    few = x[:, :, :, ::4096].contiguous()
    for m, attrs in ((64, dict()), (64, dict(normalization_term=True, ignore_nan_input=True)), (12, dict(similarity_function="L1"))):
        t, w = _parameters(m, 1, 16, 1)
        y = gpu_util.sim_ops.similarity_forward(x, t, w, blocks=[16, 1], strides=[1, 4096], padding=[14, 0], **attrs)
        want = gpu_util.sim_ops.similarity_forward(few, t, w, blocks=[16, 1], strides=[1, 1], padding=[14, 0], **attrs)
        assert float((y - want).abs().max()) <= 1e-5 * float(want.abs().max())
        dy = torch.randn(y.shape, generator=torch.Generator(device="cuda").manual_seed(3), device="cuda")
        got = gpu_util.sim_ops.similarity_parameters_grad(x, t, w, dy, blocks=[16, 1], strides=[1, 4096], padding=[14, 0], **attrs)
        want = gpu_util.sim_ops.similarity_parameters_grad(few, t, w, dy, blocks=[16, 1], strides=[1, 1], padding=[14, 0], **attrs)
        for a, b in zip(got, want):
            assert float((a - b).norm()) <= 1e-5 * float(b.norm())


@pytest.mark.parametrize("m,attrs", [(32, dict()), (5, dict(normalization_term=True)), (32, dict(similarity_function="L1"))], ids=["l2", "l2n", "l1"])
def test_forward_of_offsets_beyond_31_bits(m, attrs):
    """The sample of the parameter gradients' test, through the default dispatch of the forward pass."""
    x, (t, w) = _sample(1, 33, 8200, 8200), _parameters(m, 33, 1, 1)
    y = gpu_util.sim_ops.similarity_forward(x, t, w, blocks=[1, 1], strides=[64, 64], padding=[0, 0], **attrs)
    want = gpu_util.sim_ops.similarity_forward(x[:, :, ::64, ::64].contiguous(), t, w, blocks=[1, 1], strides=[1, 1], padding=[0, 0], **attrs)
    assert float((y - want).abs().max()) <= 1e-5 * float(want.abs().max())
