"""What surrounds the native gradient nodes: forward-mode differentiation is refused, torch.jit.trace records the calls, hooks
on saved tensors see everything a node keeps."""
import importlib

import pytest
import torch
import torch.autograd.forward_ad as forward_ad

from simnets_tf_b200 import keras
from simnets_tf_b200.ops.loss import softmax_cross_entropy
from simnets_tf_b200.simnet import SPECS, SimNet

mex_ops = importlib.import_module("simnets_tf_b200.ops.mex")
sim_ops = importlib.import_module("simnets_tf_b200.ops.similarity")
pytestmark = pytest.mark.gpu

MEX = dict(blocks=[4, 1, 1], strides=[4, 1, 1], softmax_mode=True, use_unshared_regions=False, shared_offset_region=[-1])


class Op(torch.nn.Module):
    """One operator with parameters of its own."""

    def __init__(self, call, *params):
        super().__init__()
        self.call = call
        self.params = torch.nn.ParameterList([torch.nn.Parameter(p) for p in params])

    def forward(self, x):
        return self.call(x, *self.params)


def _operators():
    gen = torch.Generator(device="cuda").manual_seed(3)

    def normal(*shape):
        return torch.randn(shape, generator=gen, device="cuda")

    labels = torch.randint(0, 7, (6,), generator=gen, device="cuda")
    off = normal(1, 8, 4, 1, 1)
    return dict(
        similarity=(Op(lambda x, t, w: sim_ops.similarity(x, t, w, blocks=[3, 3], strides=[1, 1], padding=[1, 1]), normal(8, 4, 3, 3), normal(8, 4, 3, 3).abs() + 0.1),
                    normal(6, 4, 8, 8)),
        mex=(Op(lambda x, o: mex_ops.mex(x, o, 8, **MEX), off), normal(6, 4, 8, 8)),
        mex_pooled=(Op(lambda x, o: mex_ops.mex_sum_pool2(x, o, 8, **MEX), off), normal(6, 4, 8, 8)),
        mex_pooled_f64=(Op(lambda x, o: mex_ops.mex_sum_pool2(x, o, 8, **MEX), off.double()), normal(6, 4, 8, 8).double()),
        cross_entropy=(Op(lambda x: softmax_cross_entropy(x, labels, 0.5)), normal(6, 7)))


OPERATORS = ["similarity", "mex", "mex_pooled", "mex_pooled_f64", "cross_entropy"]


@pytest.mark.parametrize("name", OPERATORS)
def test_tangents_are_refused(name):
    op, x = _operators()[name]
    for wanted in (False, True):
        with forward_ad.dual_level():
            dual = forward_ad.make_dual(x.clone().requires_grad_(wanted), torch.ones_like(x))
            with pytest.raises(NotImplementedError):
                op(dual)


def _gradients(op, x):
    x = x.clone().requires_grad_()
    y = op(x)
    dy = torch.linspace(-1, 1, y.numel(), dtype=y.dtype, device="cuda").reshape(y.shape)
    return (y.detach(),) + torch.autograd.grad(y, [x] + list(op.parameters()), dy)


@pytest.mark.parametrize("name", OPERATORS)
def test_a_recorded_call_runs_again_on_other_inputs(name):
    op, x = _operators()[name]
    traced = torch.jit.trace(op, (x,), check_trace=False)
    inputs = [x, 0.5 * x] + ([x[:4] - 1] if name != "cross_entropy" else [])         # (the labels belong to six rows)
    for v in inputs:
        for ours, ref in zip(_gradients(traced, v), _gradients(op, v)):
            assert torch.equal(ours, ref)


def test_a_recorded_network_runs_again_on_other_inputs():
    net = SimNet(SPECS["cfg3"], seed=1)
    x = torch.rand(3, 1, 28, 28, device="cuda") - 0.5
    traced = torch.jit.trace(net, (x,), check_trace=False)
    for v in (x, x * 0.5, torch.rand(5, 1, 28, 28, device="cuda") - 0.5):
        assert torch.allclose(traced(v), net(v), rtol=1e-6, atol=1e-6)


@pytest.mark.parametrize("name", OPERATORS)
def test_hooks_see_every_saved_tensor(name):
    op, x = _operators()[name]
    seen = []
    x = x.clone().requires_grad_()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: seen.append(t.shape) or t.cpu(), lambda t: t.cuda()):
        y = op(x)
    g = torch.autograd.grad(y.sum(), [x] + list(op.parameters()))
    want = {"similarity": [x.shape] + [p.shape for p in op.params], "cross_entropy": [x.shape]}.get(name, [x.shape, op.params[0].shape if len(op.params) else None, (6, 8, 8, 8)])
    assert seen == want
    for ours, ref in zip(g, torch.autograd.grad(op(x).sum(), [x] + list(op.parameters()))):
        assert torch.equal(ours, ref)


def test_a_layer_of_a_recorded_graph_takes_its_bucket_gradient_through_autograd():
    from simnets_tf_b200 import dp
    layer = keras.Mex(8, blocks=[4, 1, 1], strides=[4, 1, 1], softmax_mode=True, normalize_offsets=True, use_unshared_regions=False)
    x = torch.randn(6, 4, 8, 8, device="cuda")
    layer(x)
    bucket = dp.GradBucket(layer.parameters())
    layer(x).square().sum().backward()
    want = bucket.flat.clone()
    traced = torch.jit.trace(layer, (x,), check_trace=False)
    bucket.zero()
    traced(x).square().sum().backward()
    assert torch.allclose(bucket.flat, want, rtol=1e-6, atol=1e-6 * float(want.abs().max()))
