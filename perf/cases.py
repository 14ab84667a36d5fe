"""What this framework is timed on: passes through its public entry points, over the range of sizes, types and options that
its users have it run.

    listed()            the cases that are always timed
    draw(rng)           one more case of the same ranges
    prepare(case, seed) inputs, parameters and layers of one case, on the GPU
    run(state)          one pass through the public entry points, returning everything it computes
    work(case)          bytes and floating-point operations that a pass cannot do without
    tolerance(case)     how far another correct implementation of the same precision may be

Kinds of a case:

    classify    logits of a SimNet, no gradients (serving)
    train       loss and every parameter gradient of a SimNet, through autograd (`net.loss(...).backward()`)
    step        the same through `dp.OverlappedStep`, the captured data-parallel step, with its gradient bucket
    similarity  the `similarity` operator, forward and all three gradients
    mex         a `Mex` layer, forward and both gradients
    mixture     one EM update of the unsupervised initialisation of a Similarity layer

A SimNet here is the architecture of the two example networks (`simnets_tf_b200.netspec.SPECS`): a Similarity layer, stages
of [MEX over the channels of each pixel, doubling them, regions unshared 2 x 2; 2x2 sum pooling], a MEX over what is left
with one instance per class, softmax cross-entropy.
"""
import math

import torch

from simnets_tf_b200 import dp, keras, unsupervised
from simnets_tf_b200.ops.similarity import similarity
from simnets_tf_b200.simnet import SimNet

NAN = float("nan")
CLASSES = 10


# ------------------------------------------------------------------------------------------------------------- the cases
def _net(kind, style, batch, final, stages, templates, f64=False):
    """style "stride2": 2x2 blocks, stride 2, NaN padding 2, missing-data aware (the 1x28x28 example network);
    "same": 3x3 blocks, stride 1, padding 1 (the 3x32x32 network).  final: height and width in front of the last MEX."""
    return dict(kind=kind, style=style, batch=batch, final=final, stages=stages, templates=templates, f64=f64)


def _sim(batch, channels, height, width, templates, block_h, block_w, stride_h, stride_w, pad_h, pad_w, l1, norm, missing):
    return dict(kind="similarity", batch=batch, channels=channels, height=height, width=width, templates=templates, block_h=block_h,
                block_w=block_w, stride_h=stride_h, stride_w=stride_w, pad_h=pad_h, pad_w=pad_w, l1=l1, norm=norm, missing=missing)


def _mex(batch, channels, height, width, instances, block_c, block_h, block_w, stride_h, stride_w, pad, region, epsilon, normalize):
    """region: 0 = one offsets table shared by all positions, n = unshared n x n regions."""
    return dict(kind="mex", batch=batch, channels=channels, height=height, width=width, instances=instances, block_c=block_c, block_h=block_h,
                block_w=block_w, stride_h=stride_h, stride_w=stride_w, pad=pad, region=region, epsilon=epsilon, normalize=normalize)


def _mixture(batch, channels, height, width, templates, block, stride):
    return dict(kind="mixture", batch=batch, channels=channels, height=height, width=width, templates=templates, block=block, stride=stride)


def listed():
    return [
        # one image through the 1x28x28 example network: the smallest call there is, all latency
        dict(_net("classify", "stride2", 1, 1, 4, 32), name="classify one image"),
        # bulk evaluation with the 3x32x32 network, the last batch of a data set that no power of two divides
        dict(_net("classify", "same", 1357, 4, 3, 64), name="classify a set"),
        # an ordinary training step of the example network (its own batch size)
        dict(_net("train", "stride2", 256, 1, 4, 32), name="train small net"),
        # an ordinary training step of the deeper network, whole batch on one GPU: the largest network step
        dict(_net("train", "same", 2048, 4, 3, 64), name="train deep net"),
        # what one of eight GPUs does of that step in data-parallel training, captured
        dict(_net("step", "same", 256, 4, 3, 64), name="data-parallel share"),
        # double precision, as the gradient checks and the operators' own tests use it
        dict(_net("train", "same", 12, 4, 3, 64, f64=True), name="train in float64"),
        # a wide inner layer on data with missing entries: by far the most arithmetic
        dict(_sim(256, 64, 32, 32, 256, 3, 3, 1, 1, 1, 1, False, True, True), name="similarity missing data"),
        # L1, rectangular blocks, strides, padding and sizes that divide nothing
        dict(_sim(37, 19, 45, 37, 100, 5, 3, 2, 1, 2, 0, True, False, False), name="similarity ragged L1"),
        # a small MEX layer with unshared regions and normalised offsets
        dict(_mex(64, 32, 16, 16, 64, 32, 1, 1, 1, 1, 0, 2, 1.0, True), name="mex small unshared"),
        # a wide MEX layer whose blocks tile channels and rows and share one table: the most memory traffic
        dict(_mex(256, 256, 32, 32, 256, 4, 2, 2, 2, 2, 0, 0, 0.5, False), name="mex wide shared"),
        # overlapping, padded spatial blocks on an odd-sized map
        dict(_mex(24, 12, 41, 40, 24, 12, 3, 3, 1, 1, 1, 2, 1.0, True), name="mex overlapping blocks"),
        # one EM update of the unsupervised initialisation of the 3x32x32 network's first layer
        dict(_mixture(512, 3, 32, 32, 64, 3, 1), name="mixture update"),
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


# A drawn case stays below these, which the largest listed case of its kind reaches or nearly reaches.
_MOST_FLOPS = {"classify": 1.0e11, "train": 3.0e11, "step": 6.0e10, "f64": 3.0e9, "similarity": 4.0e11, "mex": 2.0e11, "overlapping": 1.0e10,
               "mixture": 1.0e10}


def _within(rng, make, most, largest, smallest=1):
    """make(batch) with the batch spread over smallest..largest, or up to as many as the limit allows."""
    one = work(make(1))["flops"]
    return make(_log(rng, smallest, max(smallest, min(largest, int(most / one)))))


def draw(rng):
    kind = rng.choice(["classify", "train", "train", "step", "similarity", "similarity", "mex", "mex", "mixture"])
    if kind in ("classify", "train", "step"):
        style = rng.choice(["stride2", "same"])
        stages = rng.randint(2, 4)
        final = rng.randint(1, {2: 6, 3: 4, 4: 2}[stages])
        templates = _log(rng, 12, 96 if stages < 4 else 40)
        f64 = kind == "train" and rng.random() < 0.25
        return _within(rng, lambda b: _net(kind, style, b, final, stages, templates, f64), _MOST_FLOPS["f64" if f64 else kind],
                       64 if f64 else 256 if kind == "step" else 2048)
    if kind == "similarity":
        bh, bw = rng.randint(1, 5), rng.randint(1, 5)
        l1 = rng.random() < 0.35
        norm = not l1 and rng.random() < 0.6
        args = (_log(rng, 1, 64), _log(rng, 8, 64), _log(rng, 8, 64), _log(rng, 8, 256), bh, bw, rng.randint(1, 2), rng.randint(1, 2),
                rng.randint(0, bh // 2), rng.randint(0, bw // 2), l1, norm, norm and rng.random() < 0.7)
        return _within(rng, lambda b: _sim(b, *args), _MOST_FLOPS[kind], 256)
    if kind == "mex":
        form = rng.choice(["pixel", "tiling", "overlapping"])
        if form == "pixel":             # over the channels of each pixel, regions unshared n x n
            c = _log(rng, 8, 256)
            args = (c, _log(rng, 2, 32), _log(rng, 2, 32), _log(rng, 16, 512), c, 1, 1, 1, 1, 0, rng.choice([0, 2, 2]), 1.0, True)
        elif form == "tiling":          # disjoint blocks of a few channels, rows and columns
            bc, bh = _log(rng, 1, 8), rng.choice([1, 2, 3, 4])
            args = (bc * _log(rng, 1, 64), bh * rng.randint(2, 12), bh * rng.randint(2, 12), _log(rng, 8, 256), bc, bh, bh, bh, bh, 0,
                    rng.choice([0, 0, 2]), rng.choice([0.5, 1.0]), rng.random() < 0.5)
        else:                           # every position, padded
            c, k = _log(rng, 3, 24), rng.choice([2, 3, 5])
            args = (c, rng.randint(8, 41), rng.randint(8, 41), _log(rng, 4, 32), c, k, k, 1, 1, k // 2, rng.choice([0, 2]), 1.0, True)
        return _within(rng, lambda b: _mex(b, *args), _MOST_FLOPS["overlapping" if form == "overlapping" else kind], 256)
    block = rng.randint(1, 5)
    args = (rng.choice([1, 3, 3, 8]), rng.randint(14, 40), rng.randint(14, 40), _log(rng, 8, 96), block, rng.randint(1, min(block, 2)))
    return _within(rng, lambda b: _mixture(b, *args), _MOST_FLOPS[kind], 512, 8)


# ---------------------------------------------------------------------------------------------------------------- inputs
def _layer_sizes(case):
    """(image side, [channels, side] in front of each MEX stage, channels in front of the last MEX)."""
    out = case["final"] << case["stages"]
    image = 2 * out - 4 if case["style"] == "stride2" else out
    stages = [(case["templates"] << i, out >> i) for i in range(case["stages"])]
    return image, stages, case["templates"] << case["stages"]


def _spec(case):
    image, stages, last = _layer_sizes(case)
    if case["style"] == "stride2":
        first = dict(num_instances=case["templates"], similarity_function="L2", blocks=[2, 2], strides=[2, 2], padding=[2, 2],
                     normalization_term=True, ignore_nan_input=True, out_of_bounds_value=NAN)
    else:
        first = dict(num_instances=case["templates"], similarity_function="L2", blocks=[3, 3], strides=[1, 1], padding=[1, 1])
    layers = [("similarity", first)]
    for c, _ in stages:
        layers += [("mex", dict(num_instances=2 * c, blocks=[c, 1, 1], strides=[c, 1, 1], softmax_mode=True, normalize_offsets=True,
                                use_unshared_regions=True, unshared_offset_region=[2])), ("sumpool", 2)]
    whole = [last, case["final"], case["final"]]
    layers += [("mex", dict(num_instances=CLASSES, blocks=whole, strides=whole, softmax_mode=True, normalize_offsets=True,
                            use_unshared_regions=True, shared_offset_region=[1])), ("flatten",)]
    return dict(input_shape=(_image_channels(case), image, image), classes=CLASSES, layers=layers)


def _image_channels(case):
    return 1 if case["style"] == "stride2" else 3


def _prepare_net(case, seed, gen):
    dtype = torch.float64 if case["f64"] else torch.float32
    net = SimNet(_spec(case), seed=seed % (1 << 31), device="cuda", dtype=dtype)
    # A network that has learned something: templates that look like patches of the data, weights that tell them apart and
    # log-weights spread over a few nats.  (With the near-uniform initial ones every class gets almost the same logit, and
    # the gradients are rounding errors of sums that cancel.)
    with torch.no_grad():
        for m in net.stages:
            if isinstance(m, keras.Similarity):
                m.templates.copy_(torch.rand(m.templates.shape, generator=gen, device="cuda") - 0.5)
                taps = m.sweights[0].numel()
                m.sweights.copy_(100.0 / taps * (1.0 + 0.1 * torch.randn(m.sweights.shape, generator=gen, device="cuda")))
            else:
                m.offsets.copy_(4.0 * torch.randn(m.offsets.shape, generator=gen, device="cuda"))
    image = _layer_sizes(case)[0]
    x = (torch.rand((case["batch"], _image_channels(case), image, image), generator=gen, device="cuda") - 0.5).to(dtype)
    labels = torch.randint(0, CLASSES, (case["batch"],), generator=gen, device="cuda")
    return net, x, labels


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape):
        return torch.randn(shape, generator=gen, device="cuda")

    kind = case["kind"]
    if kind in ("classify", "train", "step"):
        net, x, labels = _prepare_net(case, seed, gen)
        state = dict(kind=kind, net=net, x=x, labels=labels)
        if kind == "step":
            state["bucket"] = dp.GradBucket(net.parameters())
            state["stepper"] = dp.OverlappedStep(net, state["bucket"], x, labels, case["batch"])
        return state
    shape = (case["batch"], case["channels"], case["height"], case["width"])
    if kind == "similarity":
        x = normal(*shape)
        if case["missing"]:
            x[torch.rand(shape, generator=gen, device="cuda") < 0.2] = NAN
        blocks = [case["block_h"], case["block_w"]]
        t = 0.1 * normal(case["templates"], case["channels"], *blocks)
        w = (1.0 + 0.1 * normal(*t.shape)).abs() + 1e-3
        attrs = dict(similarity_function="L1" if case["l1"] else "L2", blocks=blocks, strides=[case["stride_h"], case["stride_w"]],
                     padding=[case["pad_h"], case["pad_w"]], normalization_term=case["norm"], ignore_nan_input=case["missing"])
        oh, ow = _sim_out(case)
        return dict(kind=kind, x=x.requires_grad_(), t=t.requires_grad_(), w=w.requires_grad_(), attrs=attrs,
                    dy=normal(case["batch"], case["templates"], oh, ow))
    if kind == "mex":
        region = dict(use_unshared_regions=False, shared_offset_region=[-1]) if case["region"] == 0 else dict(
            use_unshared_regions=True, unshared_offset_region=[case["region"]])
        layer = keras.Mex(case["instances"], padding=[0, case["pad"], case["pad"]], strides=[case["block_c"], case["stride_h"], case["stride_w"]],
                          blocks=[case["block_c"], case["block_h"], case["block_w"]], epsilon=case["epsilon"], softmax_mode=True,
                          normalize_offsets=case["normalize"], offsets_initializer="zeros", **region)
        layer.build(shape, torch.device("cuda"), torch.float32)
        with torch.no_grad():
            layer.offsets.copy_(normal(*layer.offsets.shape))
        co, oh, ow = _mex_out(case)
        return dict(kind=kind, layer=layer, x=normal(*shape).requires_grad_(), dy=normal(case["batch"], case["instances"] * co, oh, ow))
    est = unsupervised.DiagonalGMM([case["block"]] * 2, [case["stride"]] * 2, case["templates"], seed=seed % (1 << 31))
    x = torch.rand(shape, generator=gen, device="cuda") - 0.5
    est.init(x)
    return dict(kind=kind, est=est, x=x)


# -------------------------------------------------------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "classify":
        with torch.no_grad():
            return state["net"](state["x"])
    if kind == "train":
        net = state["net"]
        net.zero_grad(set_to_none=True)
        loss = net.loss(state["x"], state["labels"])
        loss.backward()
        return [loss.detach()] + [p.grad for p in net.parameters()]
    if kind == "step":
        loss = state["stepper"].run()
        return [loss.detach()] + [p.grad for p in state["net"].parameters()]
    if kind == "similarity":
        x, t, w = state["x"], state["t"], state["w"]
        y = similarity(x, t, w, **state["attrs"])
        return (y.detach(),) + torch.autograd.grad(y, (x, t, w), state["dy"])
    if kind == "mex":
        x, layer = state["x"], state["layer"]
        y = layer(x)
        return (y.detach(),) + torch.autograd.grad(y, (x, layer.offsets), state["dy"])
    return state["est"].update(state["x"])


# ------------------------------------------------------------------------------------------------------------------ work
def _sim_out(case):
    return ((case["height"] + 2 * case["pad_h"] - case["block_h"]) // case["stride_h"] + 1,
            (case["width"] + 2 * case["pad_w"] - case["block_w"]) // case["stride_w"] + 1)


def _mex_out(case):
    return (case["channels"] // case["block_c"], (case["height"] + 2 * case["pad"] - case["block_h"]) // case["stride_h"] + 1,
            (case["width"] + 2 * case["pad"] - case["block_w"]) // case["stride_w"] + 1)


def work(case):
    """Bytes: inputs and parameters once, results once (activations between the layers of a network do not count).
    Operations: a Similarity term w f(x - t) is a difference, a product and a multiply-add (4) in the forward pass and in the
    input gradient, a difference, two products and two multiply-adds (7) in the parameter gradients; a MEX term is one
    multiply-add (2) in each of its three passes, its exponentials not counted."""
    kind, b = case["kind"], case["batch"]
    if kind in ("classify", "train", "step"):
        size = 8 if case["f64"] else 4
        image, stages, last = _layer_sizes(case)
        taps = _image_channels(case) * (4 if case["style"] == "stride2" else 9)
        params = 2 * case["templates"] * taps + sum(4 * 2 * c * c for c, _ in stages) + CLASSES * last * case["final"] ** 2
        sim = case["templates"] * taps * stages[0][1] ** 2
        mex = sum(2 * c * c * s * s for c, s in stages) + CLASSES * last * case["final"] ** 2
        x = b * _image_channels(case) * image * image
        if kind == "classify":
            return dict(bytes=size * (x + params + b * CLASSES), flops=b * (4.0 * sim + 2.0 * mex))
        return dict(bytes=size * (x + 2 * params) + 8 * b, flops=b * (11.0 * sim + 6.0 * mex))
    x = b * case["channels"] * case["height"] * case["width"]
    if kind == "similarity":
        oh, ow = _sim_out(case)
        params = case["templates"] * case["channels"] * case["block_h"] * case["block_w"]
        y = b * case["templates"] * oh * ow
        return dict(bytes=4.0 * (2 * x + 4 * params + 2 * y), flops=15.0 * y * (params // case["templates"]))
    if kind == "mex":
        co, oh, ow = _mex_out(case)
        taps = case["block_c"] * case["block_h"] * case["block_w"]
        y = b * case["instances"] * co * oh * ow
        params = max(1, case["region"]) ** 2 * case["instances"] * taps
        return dict(bytes=4.0 * (2 * x + 2 * params + 2 * y), flops=6.0 * y * taps)
    taps = case["channels"] * case["block"] ** 2
    oh, ow = ((n - case["block"]) // case["stride"] + 1 for n in (case["height"], case["width"]))
    return dict(bytes=4.0 * (x + 4 * case["templates"] * taps), flops=11.0 * b * oh * ow * case["templates"] * taps)


def tolerance(case):
    """Sums of 32-bit terms in another order: about 1e-5 of a tensor's norm.  A network's parameter gradients have passed
    through up to six layers and through the offsets' normalisation, whose gradient subtracts what a row has in common, so
    that a rounding in one layer comes out some hundred times larger."""
    kind = case["kind"]
    if kind == "classify":
        return {"rel": 1e-5}
    if kind in ("train", "step"):
        return {"rel": 1e-9 if case["f64"] else 2e-3}
    if kind == "mixture":
        return {"rel": 1e-4}
    return {"rel": 2e-5, "max": 2e-3}
