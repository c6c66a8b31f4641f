"""The extension's ops as one `torch.autograd.Function`, for the two callers that see a Function but not a node made in C++:
`torch.jit.trace` records a Function's call (the extension allocates outside the dispatcher: to a trace its results are
constants), and forward-mode differentiation refuses a Function without a jvp (a node made in C++ drops the tangent, which
then counts as zero)."""
from __future__ import annotations

import torch
from torch.autograd import forward_ad


def active():
    return forward_ad._current_level >= 0 or torch._C._get_tracing_state() is not None


class _Recorded(torch.autograd.Function):
    @staticmethod
    def forward(ctx, op, *args):
        ctx.op = op
        ctx.args = [None if isinstance(a, torch.Tensor) else a for a in args]
        ctx.at = [i for i, a in enumerate(args) if isinstance(a, torch.Tensor)]
        ctx.save_for_backward(*(args[i] for i in ctx.at))
        return op(*args)

    @staticmethod
    def backward(ctx, *cotangents):
        args, leaves = list(ctx.args), []
        with torch.enable_grad():
            for i, t in zip(ctx.at, ctx.saved_tensors):
                args[i] = t.detach()
                if ctx.needs_input_grad[1 + i]:
                    leaves.append((i, args[i].requires_grad_()))
            out = ctx.op(*args)
        pairs = [(o, c) for o, c in zip(out if isinstance(out, tuple) else (out,), cotangents) if o is not None and c is not None]
        grads = [None] * (1 + len(args))
        for (i, _), g in zip(leaves, torch.autograd.grad([o for o, _ in pairs], [t for _, t in leaves], [c for _, c in pairs],
                                                         allow_unused=True)):
            grads[1 + i] = g
        return tuple(grads)


def call(op, *args):
    return _Recorded.apply(op, *args) if active() else op(*args)
