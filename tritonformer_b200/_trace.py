"""The operators under torch.jit.trace.

A call of the native host path leaves nothing in a graph but the allocation of its result, so while a trace is being recorded
the module hands its calls to `record`, which makes each of them one autograd Function: a node that the traced graph replays.
"""
import contextlib

import torch
from torch.autograd import Function

from . import _host


@contextlib.contextmanager
def _not_recording():
    state = torch._C._get_tracing_state()
    torch._C._set_tracing_state(None)
    try:
        yield state is not None
    finally:
        torch._C._set_tracing_state(state)


class NativeCall(Function):
    """call(*args), with a backward that runs the backward of the call's own graph."""

    @staticmethod
    def forward(ctx, call, *args):
        tensors = [i for i, a in enumerate(args) if isinstance(a, torch.Tensor)]
        inner = list(args)
        with _not_recording() as recording:
            with torch.set_grad_enabled(any(ctx.needs_input_grad)):
                for i in tensors:
                    inner[i] = args[i].detach().requires_grad_(ctx.needs_input_grad[i + 1])
                out = call(*inner)
            ctx.graph = (out, [inner[i] for i in tensors], tensors, len(args))
            value, shape, strides = out.detach(), tuple(out.shape), out.stride()
        if not recording:
            return value
        # recorded, because the graph has to know where the output comes from
        result = torch.empty_strided(shape, strides, device=value.device, dtype=value.dtype)
        with _not_recording():
            return result.copy_(value)

    @staticmethod
    def backward(ctx, grad_output):
        out, inner, at, count = ctx.graph
        wanted = [(i, t) for i, t in zip(at, inner) if t.requires_grad]
        grads = torch.autograd.grad(out, [t for _, t in wanted], grad_output, retain_graph=True, allow_unused=True)
        result = [None] * count
        for (i, _), g in zip(wanted, grads):
            result[i] = g
        return (None, *result)


def record(call, *args):
    return NativeCall.apply(call, *args)


_host.set_recorder(record)
