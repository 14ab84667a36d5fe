"""`mex` and its gradient ops, with the signature of the reference's python wrapper
(HUJI-Deep/simnets-tf python/simnets/ops/mex.py:114-195), its `_mex_dims_helper` (:17-38),
`_expand_dim_specification` (:84-112) and the gradient wiring of `_mex_grad` (:47-81).
"""
import ctypes as C

import torch

from .. import _lib, abi
from .. import _torch_glue
from .._torch_glue import dtype_code, require_cuda, sequence_key, stream_ptr

_DEFAULTS = dict(softmax_mode=False, padding=[0, 0, 0], strides=[1, 1, 1], blocks=[1, 1, 1], epsilon=1.0,
                 blocks_out_of_bounds_value=0.0, blocks_round_down=True, use_unshared_regions=True,
                 shared_offset_region=[-1], unshared_offset_region=[-1])


def _attrs(**given):
    """Op attrs with the op registration's defaults (reference src/ops/mex_op.cpp:58-74) for every None."""
    out = dict(_DEFAULTS)
    for k, v in given.items():
        if v is not None:
            out[k] = v
    return out


def _mex_dims_helper(input_dim, num_instances, blocks, padding=[0], strides=[1], blocks_round_down=True,
                     use_unshared_regions=True, shared_offset_region=[-1], unshared_offset_region=[-1]):
    """Number of offset regions for an input of shape `input_dim` = [C, H, W] (or -1 if invalid)."""
    args = []

    def add_array(l):
        l = [int(e) for e in l]
        args.extend([C.c_int(len(l)), (C.c_int * len(l))(*l)])

    add_array(input_dim)
    add_array(padding)
    add_array(strides)
    args.extend([C.c_int(num_instances), C.c_int(blocks_round_down), C.c_int(use_unshared_regions)])
    add_array(blocks)
    add_array(shared_offset_region)
    add_array(unshared_offset_region)
    return _lib.lib().get_mex_offsets_nregions(*args)


def _expand_dim_specification(image_shape, dim_spec):
    """Expand a 2- or 3-long dimension specification: prepend -1 to a pair, then replace every -1
    with the corresponding image dimension (`image_shape` has 3 entries, or 4 with the batch)."""
    if len(dim_spec) != 2 and len(dim_spec) != 3:
        raise ValueError('Bad dimensions specifications, should be a list of two or three, got %s' % dim_spec)
    image_shape = list(image_shape)
    if len(image_shape) == 3:
        image_shape = [None] + image_shape
    dim_spec = list(dim_spec)
    if len(dim_spec) == 2:
        dim_spec = [-1] + dim_spec
    for i in range(3):
        if dim_spec[i] == -1:
            dim_spec[i] = image_shape[i + 1]
    return dim_spec


def _desc_of(shape, dtype, num_instances, attrs, flags=0):
    if len(shape) != 4:
        raise ValueError("input must be 4-D")
    return abi.make_mex_desc(shape, num_instances, attrs["softmax_mode"], attrs["padding"], attrs["strides"],
                             attrs["blocks"], attrs["epsilon"], attrs["blocks_out_of_bounds_value"], attrs["blocks_round_down"],
                             attrs["use_unshared_regions"], attrs["shared_offset_region"], attrs["unshared_offset_region"],
                             dtype=abi.F32 if dtype == torch.float32 else abi.F64, flags=flags | _torch_glue.DEFAULT_FLAGS)


def _desc(input, num_instances, attrs, flags=0):
    dtype_code(input)           # (rejects anything but float32 / float64)
    return _desc_of(tuple(input.shape), input.dtype, num_instances, attrs, flags)


def _geometry(d):
    g = abi.MexGeometry()
    _lib.check(_lib.lib().simnets_mex_dims(C.byref(d), C.byref(g)))
    return g


_PLANS = _torch_glue.PlanCache()


def mex_plan(shape, dtype, num_instances, attrs):
    """The native plan of this input shape, type and attributes (a complete dict, see `_attrs`)."""
    key = (shape, dtype, num_instances, _torch_glue.DEFAULT_FLAGS) + tuple(map(sequence_key, attrs.values()))
    return _PLANS.get(key, lambda: _lib.ops().MexPlan(bytes(_desc_of(tuple(shape), dtype, num_instances, attrs))))


def _plan_of(input, num_instances, attrs):
    dtype_code(input)           # (rejects anything but float32 / float64)
    return mex_plan(input.shape, input.dtype, num_instances, attrs)


def mex_layer_workspace(input, num_instances, pooled=False, flags=0, **attrs):
    """A workspace of one layer's own, large enough for its forward and gradient calls: give it to `mex_forward`
    as `workspace=` and to the gradient ops as `primed_workspace=`, and they reuse the per-position maxima and
    the offsets tables of the forward pass instead of computing them again."""
    return mex_layer_workspace_for(tuple(input.shape), input.dtype, require_cuda(input), num_instances, pooled=pooled, flags=flags, **attrs)


def mex_layer_workspace_for(input_shape, dtype, device, num_instances, pooled=False, flags=0, **attrs):
    """`mex_layer_workspace` for an input that does not exist yet (shape, dtype and device given)."""
    return mex_plan(tuple(input_shape), dtype, num_instances, _attrs(**attrs)).layer_workspace(flags, pooled, torch.device(device))


def mex_workspace_maxima(input_shape, dtype, num_instances, workspace, flags=0, **attrs):
    """Device address inside `workspace` (a tensor from `mex_layer_workspace`) where the forward pass of this layer reads the
    per-position extrema of its patches, or None for shapes that find them on the fly.  A layer in front that writes them
    there (ops.similarity.similarity_forward(..., extrema=...)) lets `mex_forward(..., flags=FLAG_MEX_MAXIMA_GIVEN)` skip
    its own pass over the input; only valid when every patch is exactly the channels of one pixel."""
    return mex_plan(tuple(input_shape), dtype, num_instances, _attrs(**attrs)).maxima(flags, workspace) or None


def mex_forward(input, offsets, num_instances, flags=0, workspace=None, **attrs):
    """The `Mex` op: [batch, num_instances * channels_out, height_out, width_out].  `workspace`: a buffer from
    `mex_layer_workspace` to run in instead of scratch of the call's own."""
    return _lib.ops().mex_forward(_plan_of(input, num_instances, _attrs(**attrs)), input, offsets, flags, workspace)


def mex_forward_pool2(input, offsets, num_instances, flags=0, workspace=None, **attrs):
    """The `Mex` op and the 2x2 sum pooling of its output in one library call: (y, y_pooled).  float32, even output
    height and width.  On the pair-tile kernels the forward kernel's epilogue does the pooling."""
    return _lib.ops().mex_forward_pool2(_plan_of(input, num_instances, _attrs(**attrs)), input, offsets, flags, workspace)


def mex_input_grad(input, offsets, orig_output, output_grad, num_instances, flags=0, primed_workspace=None, pooled=False, **attrs):
    """The `MexInputGrad` op.  pooled=True: `output_grad` is the gradient of a 2x2 sum pooling of the output
    (half height and width); the library reads it in place of its 2x upsampling."""
    return _lib.ops().mex_input_grad(_plan_of(input, num_instances, _attrs(**attrs)), input, offsets, orig_output, output_grad, flags, primed_workspace, pooled)


def mex_offsets_grad(input, offsets, orig_output, output_grad, num_instances, flags=0, primed_workspace=None, out=None, pooled=False, **attrs):
    """The `MexOffsetsGrad` op.  `out` / FLAG_ACCUMULATE as in `similarity_parameters_grad`; `pooled` as in
    `mex_input_grad`."""
    return _lib.ops().mex_offsets_grad(_plan_of(input, num_instances, _attrs(**attrs)), input, offsets, orig_output, output_grad, flags, primed_workspace,
                                       pooled, out)


def mex_backward(input, offsets, orig_output, output_grad, num_instances, flags=0, primed_workspace=None, pooled=False, doff_out=None, **attrs):
    """`MexInputGrad` and `MexOffsetsGrad` in one library call: (input_grad, offsets_grad).  `pooled` as in
    `mex_input_grad`.  `primed_workspace` (all three gradient ops): the buffer that `mex_forward` ran in for the same
    input and offsets, untouched since.  With FLAG_ACCUMULATE in `flags` the offsets gradient is added to `doff_out`."""
    return _lib.ops().mex_backward(_plan_of(input, num_instances, _attrs(**attrs)), input, offsets, orig_output, output_grad, flags, primed_workspace,
                                   pooled, doff_out)


def sum_pool2x2(y):
    """2x2 / stride-2 sum pooling of a float32 CUDA tensor [B, C, H, W] with even H and W (the library's kernel)."""
    dev = require_cuda(y)
    y = y.contiguous()
    out = torch.empty(y.shape[:2] + (y.shape[2] // 2, y.shape[3] // 2), dtype=y.dtype, device=dev)
    with torch.cuda.device(dev):
        _lib.check(_lib.lib().simnets_sum_pool2x2_forward(y.shape[0] * y.shape[1], y.shape[2], y.shape[3], y.data_ptr(), out.data_ptr(),
                                                          stream_ptr(dev)))
    return out


def mex_recorded(plan_of, input, offsets, layer_ws=None, fwd_flags=0, op_flags=0, sum_pool2=False):
    """`mex_with_plan` while torch.jit.trace records, on the plan of whatever input the recorded graph gets: `plan_of(input)`.  Its
    gradients go through autograd, also to the `.grad` that a sink stands for."""
    return _torch_glue.recorded(lambda x, o: mex_with_plan(plan_of(x), x, o, layer_ws, fwd_flags, op_flags, sum_pool2), input, offsets)


def mex_with_plan(plan, input, offsets, layer_ws=None, fwd_flags=0, op_flags=0, sum_pool2=False, grad_sink=None):
    """`mex_in_workspace` on a plan the caller holds (`mex_plan`)."""
    apply = _lib.ops().mex_apply
    if sum_pool2 and (plan.height_out % 2 or plan.width_out % 2):
        return torch.nn.functional.avg_pool2d(apply(plan, input, offsets, layer_ws, fwd_flags, op_flags, False, grad_sink), 2) * 4.0
    return apply(plan, input, offsets, layer_ws, fwd_flags, op_flags, sum_pool2, grad_sink)


def mex(input, offsets, num_instances, softmax_mode=None, padding=None, strides=None, blocks=None, epsilon=None,
        blocks_out_of_bounds_value=None, blocks_round_down=None, use_unshared_regions=None, shared_offset_region=None,
        unshared_offset_region=None, name=None):
    """Computes the MEX layer given a 4-D `input` and 5-D `offsets`
    ([num_regions, num_instances, block_c, block_h, block_w]).

    Same arguments, defaults and result as the reference's `simnets.ops.mex.mex`; `name` is accepted
    and ignored.  Differentiable w.r.t. `input` and `offsets`.
    """
    attrs = _attrs(softmax_mode=softmax_mode, padding=padding, strides=strides, blocks=blocks, epsilon=epsilon,
                   blocks_out_of_bounds_value=blocks_out_of_bounds_value, blocks_round_down=blocks_round_down,
                   use_unshared_regions=use_unshared_regions, shared_offset_region=shared_offset_region,
                   unshared_offset_region=unshared_offset_region)
    return _mex(input, offsets, num_instances, attrs)


def _mex(input, offsets, num_instances, attrs, layer_ws=None, fwd_flags=0, op_flags=0, sum_pool2=False, grad_sink=None):
    if _torch_glue.is_tracing():
        return mex_recorded(lambda x: _plan_of(x, num_instances, attrs), input, offsets, layer_ws, fwd_flags, op_flags, sum_pool2)
    return mex_with_plan(_plan_of(input, num_instances, attrs), input, offsets, layer_ws, fwd_flags, op_flags, sum_pool2, grad_sink)


def mex_sum_pool2(input, offsets, num_instances, layer_ws=None, fwd_flags=0, op_flags=0, grad_sink=None, **kwargs):
    """`mex(...)` followed by a 2x2 sum pooling (the MEX + pooling pair of the reference's example networks,
    README.md:114-131, where the pooling is `4 * AveragePooling2D(2)`), with the pooling's backward folded into
    the MEX gradient kernels.  Same keyword arguments as `mex`.  Falls back to the two separate ops when the
    MEX output height or width is odd."""
    return mex_in_workspace(input, offsets, num_instances, layer_ws=layer_ws, fwd_flags=fwd_flags, op_flags=op_flags, sum_pool2=True,
                            grad_sink=grad_sink, **kwargs)


def mex_in_workspace(input, offsets, num_instances, layer_ws=None, fwd_flags=0, op_flags=0, sum_pool2=False, grad_sink=None, **kwargs):
    """`mex(...)` (or `mex_sum_pool2(...)`) with the library's extras: a layer workspace the caller made
    (`mex_layer_workspace_for`), flags for the forward call only (abi.FLAG_MEX_MAXIMA_GIVEN after the layer in front has
    filled in the extrema), flags for the forward and the gradient calls (abi.FLAG_MEX_NORMALIZED_OFFSETS: `offsets` are raw
    and the gradient comes back with respect to them), a tensor that the offsets gradient is ADDED to instead of being
    handed to autograd (`grad_sink`: the offsets' slice of a data-parallel gradient bucket)."""
    attrs = _attrs(**{k: v for k, v in kwargs.items() if k != "name"})
    return _mex(input, offsets, num_instances, attrs, layer_ws, fwd_flags, op_flags, sum_pool2, grad_sink)
