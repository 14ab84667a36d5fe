"""Plumbing between torch tensors and the library: dtype codes, the current stream, the plans of recent calls and per-op
timing."""

import torch

from . import _lib, abi

# Descriptor flags OR-ed into every op call of this process; 0 unless a program sets it (an A/B measurement that
# wants, say, abi.FLAG_MEX_NO_PAIR_TILES on every layer assigns it before the first call).
DEFAULT_FLAGS = 0


def dtype_code(t):
    if t.dtype == torch.float32:
        return abi.F32
    if t.dtype == torch.float64:
        return abi.F64
    raise TypeError("simnets ops are registered for float32 and float64 only, got %s" % t.dtype)


def require_cuda(*tensors):
    dev = tensors[0].device
    for t in tensors:
        if not t.is_cuda:
            raise RuntimeError("simnets_b200 has no CPU kernels: every tensor must live on a CUDA device")
        if t.device != dev:
            raise RuntimeError("all tensors of one op call must be on the same device")
        if t.dtype != tensors[0].dtype:
            raise TypeError("all tensors of one op call must share a dtype")
    return dev


def stream_ptr(dev):
    return torch.cuda.current_stream(dev).cuda_stream


def sequence_key(v):
    """`v` as part of a dictionary key: lists and tuples by value."""
    return tuple(v) if isinstance(v, (list, tuple)) else v


class _Recorded(torch.autograd.Function):
    """An operator call as one node of the graph that torch.jit.trace records.  The tracer sees torch's own operators only: it
    would keep the result of a native call as a constant.  As a node, the call is made again (plan, checks and gradient
    included) whenever the recorded graph runs."""

    @staticmethod
    def forward(ctx, call, *tensors):
        with torch.enable_grad():
            ctx.inputs = [t.detach().requires_grad_(wanted) for t, wanted in zip(tensors, ctx.needs_input_grad[1:])]
            ctx.output = call(*ctx.inputs)
        return ctx.output.detach()

    @staticmethod
    def backward(ctx, grad):
        wanted = [t for t in ctx.inputs if t.requires_grad]
        got = iter(torch.autograd.grad(ctx.output, wanted, grad, retain_graph=True, create_graph=torch.is_grad_enabled()))
        return (None,) + tuple(next(got) if t.requires_grad else None for t in ctx.inputs)


is_tracing = torch._C._is_tracing           # (torch.jit.is_tracing without its Python frame: every operator call asks)


def recorded(call, *tensors):
    """call(*tensors) while torch.jit.trace is recording (see `_Recorded`)."""
    return _Recorded.apply(call, *tensors)


class PlanCache(object):
    """The native plans (descriptor, geometry) of the calls seen last, by everything that determines them.  Bounded: a
    program that keeps changing shapes starts over after `limit` of them."""

    def __init__(self, limit=1024):
        self.limit, self.plans = limit, {}

    def get(self, key, make):
        try:
            plan = self.plans.get(key)
        except TypeError:                   # an attribute that cannot be hashed (an array, say): no caching
            return make()
        if plan is None:
            plan = make()
            if len(self.plans) >= self.limit:
                self.plans.clear()
            self.plans[key] = plan
        return plan


class OpProfile(object):
    """Optional per-op device timing: when enabled, every operator call is bracketed by CUDA events on
    the stream it launches on, together with the algorithmic bytes and term count of that call."""

    def start(self):
        _lib.ops().profile_start()

    def stop(self):
        """Stop recording and return {key: dict(calls, ms, bytes, terms)} (synchronises)."""
        torch.cuda.synchronize()
        out = {}
        for key, ms, nbytes, terms in _lib.ops().profile_stop():
            r = out.setdefault(key, dict(calls=0, ms=0.0, bytes=0, terms=0))
            r["calls"] += 1
            r["ms"] += ms
            r["bytes"] += int(nbytes)
            r["terms"] += int(terms)
        return out


PROFILE = OpProfile()
