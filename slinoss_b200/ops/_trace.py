"""The ops under ``torch.jit.trace``: the native path is invisible to the tracer, so a traced call goes through a Python
autograd function, which the trace records and runs again with the inputs of the traced program."""

from __future__ import annotations

import torch

tracing = torch._C._is_tracing


class _Recorded(torch.autograd.Function):
    @staticmethod
    def forward(ctx, call, *args):
        ctx.set_materialize_grads(False)
        state = torch._C._get_tracing_state()
        torch._C._set_tracing_state(None)
        try:
            with torch.enable_grad():
                ctx.leaves = [a if a is None else a.detach().requires_grad_(a.requires_grad) for a in args]
                ctx.outs = call(*ctx.leaves)
            outs = [t.detach() for t in ctx.outs]
        finally:
            torch._C._set_tracing_state(state)
        return tuple(t.detach() for t in outs)  # (results of operations that the tracer has seen)

    @staticmethod
    def backward(ctx, *grads):
        wanted = [a for a in ctx.leaves if a is not None and a.requires_grad]
        given = [(o, g) for o, g in zip(ctx.outs, grads) if g is not None]
        got = iter(torch.autograd.grad([o for o, _ in given], wanted, [g for _, g in given], allow_unused=True,
                                       retain_graph=True))
        return (None, *(next(got) if a is not None and a.requires_grad else None for a in ctx.leaves))


def recorded(call, *args):
    """``call(*args)``, a tuple of tensors of tensor (or ``None``) arguments, as one operation of the trace."""
    return _Recorded.apply(call, *args)
