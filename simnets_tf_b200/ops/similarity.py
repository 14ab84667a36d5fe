"""`similarity` and its gradient ops, with the signature of the reference's python wrapper
(HUJI-Deep/simnets-tf python/simnets/ops/similarity.py:48-121) and the gradient wiring of its
`_similarity_grad` (same file, :18-45).  Tensors are torch CUDA tensors; the work is done by the
CUDA library through the C ABI.
"""
from .. import _lib, abi
from .. import _torch_glue
from .._torch_glue import dtype_code, sequence_key

_DEFAULTS = dict(similarity_function="L2", blocks=[3, 3], strides=[2, 2], padding=[0, 0], normalization_term=False,
                 normalization_term_fudge=0.001, ignore_nan_input=False, out_of_bounds_value=0.0)


def _attrs(**given):
    """Op attrs with the op registration's defaults (reference src/ops/similarity_op.cpp:61-75) for every None."""
    out = dict(_DEFAULTS)
    for k, v in given.items():
        if v is not None:
            out[k] = v
    return out


def _desc(input, templates, weights, attrs, flags=0):
    if input.dim() != 4 or templates.dim() != 4 or weights.dim() != 4:
        raise ValueError("input, templates and weights must be 4-D")
    if templates.shape != weights.shape:
        raise ValueError("templates and weights must have the same shape")
    if templates.shape[1] != input.shape[1]:
        raise ValueError("Number of channels mismatch between input and template")
    blocks = list(attrs["blocks"])
    if list(templates.shape[2:]) != [int(b) for b in blocks]:
        raise ValueError("templates spatial shape %s does not match blocks %s" % (list(templates.shape[2:]), blocks))
    return abi.make_sim_desc(input.shape, templates.shape[0], attrs["similarity_function"], blocks, attrs["strides"],
                             attrs["padding"], attrs["normalization_term"], attrs["normalization_term_fudge"],
                             attrs["ignore_nan_input"], attrs["out_of_bounds_value"], dtype=dtype_code(input), flags=flags | _torch_glue.DEFAULT_FLAGS)


_PLANS = _torch_glue.PlanCache()


def similarity_plan(input, templates, weights, attrs):
    """The native plan of these shapes and attributes (a complete dict, see `_attrs`)."""
    key = (input.shape, input.dtype, templates.shape, weights.shape, _torch_glue.DEFAULT_FLAGS) + tuple(map(sequence_key, attrs.values()))
    return _PLANS.get(key, lambda: _lib.ops().SimPlan(bytes(_desc(input, templates, weights, attrs))))


def similarity_forward(input, templates, weights, flags=0, extrema=None, **attrs):
    """The `Similarity` op: [batch, templates, out_h, out_w].  `extrema=(max_ptr, min_ptr)`: device addresses (or None)
    that receive the per-pixel maximum / minimum of the output over the templates, float32 [batch, out_h, out_w]."""
    up, down = extrema if extrema is not None else (None, None)
    return _lib.ops().sim_forward(similarity_plan(input, templates, weights, _attrs(**attrs)), input, templates, weights, flags, up or 0, down or 0)


def similarity_input_grad(input, templates, weights, input_grad, flags=0, **attrs):
    """The `SimilarityInputGrad` op (its fourth input is the gradient w.r.t. the op's output)."""
    return _lib.ops().sim_input_grad(similarity_plan(input, templates, weights, _attrs(**attrs)), input, templates, weights, input_grad, flags)


def similarity_parameters_grad(input, templates, weights, output_grad, flags=0, out=None, **attrs):
    """The `SimilarityParametersGrad` op: (templates_grad, weights_grad).

    `out=(dt, dw)` writes into caller-owned tensors (e.g. slices of a data-parallel gradient
    bucket); with `flags & FLAG_ACCUMULATE` the results are added to them."""
    dt, dw = out if out is not None else (None, None)
    return _lib.ops().sim_params_grad(similarity_plan(input, templates, weights, _attrs(**attrs)), input, templates, weights, output_grad, flags, dt, dw)


def similarity_recorded(plan_of, input, templates, weights, flags=0, extrema=None):
    """The differentiable op while torch.jit.trace records, on the plan of whatever input the recorded graph gets: `plan_of(input,
    templates, weights)`.  Its gradients go through autograd, also to the `.grad` that a sink stands for."""
    up, down = extrema if extrema is not None else (None, None)
    return _torch_glue.recorded(lambda x, t, w: _lib.ops().sim_apply(plan_of(x, t, w), x, t, w, flags, up or 0, down or 0, None, None),
                                input, templates, weights)


def _apply(input, templates, weights, attrs, flags=0, extrema=None, grad_sinks=None):
    if _torch_glue.is_tracing():
        return similarity_recorded(lambda x, t, w: similarity_plan(x, t, w, attrs), input, templates, weights, flags, extrema)
    up, down = extrema if extrema is not None else (None, None)
    dt, dw = grad_sinks if grad_sinks is not None else (None, None)
    return _lib.ops().sim_apply(similarity_plan(input, templates, weights, attrs), input, templates, weights, flags, up or 0, down or 0, dt, dw)


def similarity(input, templates, weights, similarity_function=None, blocks=None, strides=None, padding=None,
               normalization_term=None, normalization_term_fudge=None, ignore_nan_input=None, out_of_bounds_value=None,
               name=None, ksize=None):
    """Computes a similarity measure given 4-D `input`, `templates` and `weights` tensors.

    Same arguments, defaults and result as the reference's `simnets.ops.similarity.similarity`; `name`
    is accepted and ignored, `ksize` is an alias of `blocks` (the name the reference's README uses).
    Differentiable w.r.t. all three tensors.
    """
    if blocks is None and ksize is not None:
        blocks = ksize
    attrs = _attrs(similarity_function=similarity_function, blocks=blocks, strides=strides, padding=padding,
                   normalization_term=normalization_term, normalization_term_fudge=normalization_term_fudge,
                   ignore_nan_input=ignore_nan_input, out_of_bounds_value=out_of_bounds_value)
    return _apply(input, templates, weights, attrs)


def similarity_of_raw_weights(input, templates, raw_weights, flags=0, extrema=None, grad_sinks=None, **attrs):
    """`similarity(input, templates, abs(raw_weights), ...)`, differentiable w.r.t. all three tensors, with the absolute
    value and its gradient taken inside the library's kernels (abi.FLAG_SIM_ABS_WEIGHTS): what the reference's Keras
    layer computes with `K.abs(self.sweights)` in front of the op (python/simnets/keras.py:65)."""
    return _apply(input, templates, raw_weights, _attrs(**attrs), flags | abi.FLAG_SIM_ABS_WEIGHTS, extrema, grad_sinks)
