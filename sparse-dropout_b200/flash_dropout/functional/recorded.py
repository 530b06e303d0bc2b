"""Native operators inside ``torch.jit.trace``.

The extension (csrc/sd_torch.cpp) makes its results outside the dispatcher, so a trace would take them for constants and
answer every later input with the example's result.  While a trace is recorded the operators go through ``recorded``, which
a trace holds as one operation: it runs the call again, with fresh masks and with its gradients, whenever the trace runs.
"""
from __future__ import annotations

import torch


class _Recorded(torch.autograd.Function):
    @staticmethod
    def forward(ctx, call, *tensors):
        state = torch._C._get_tracing_state()
        torch._C._set_tracing_state(None)          # the call itself is not recorded, and sees no trace
        try:
            with torch.enable_grad(), torch.autocast("cuda", enabled=False):
                leaves = [t.detach().requires_grad_(needed) for t, needed in zip(tensors, ctx.needs_input_grad[1:])]
                out = call(*leaves)
            value = out.detach()
        finally:
            torch._C._set_tracing_state(state)
        ctx.leaves, ctx.out = leaves, out
        result = torch.empty(0, dtype=out.dtype, device=out.device)    # a tensor that the trace knows,
        result.data = value                                             # with the call's result for its memory
        return result

    @staticmethod
    def backward(ctx, dy):
        wanted = [t for t in ctx.leaves if t.requires_grad]
        grads = iter(torch.autograd.grad(ctx.out, wanted, dy, retain_graph=True, allow_unused=True))
        return (None, *(next(grads) if t.requires_grad else None for t in ctx.leaves))


def recorded(operator, tensors, *rest):
    """``operator(*tensors, *rest)`` as one operation of the trace that is being recorded.  Under autocast the tensors are
    cast here, by operators that the trace sees."""
    if torch.is_autocast_enabled("cuda"):
        tensors = [t.to(torch.get_autocast_dtype("cuda")) for t in tensors]
    return _Recorded.apply(lambda *new: operator(*new, *rest), *tensors)
