"""An op of the native extension as ONE Python autograd function, for the callers that need to see one.

The extension builds its backward nodes in C++, where a tracer records nothing and forward-mode tangents or functorch
levels would pass by without a word.  In those contexts its entry points come here instead: ``torch.jit.trace`` gets a
node that runs the op again, and forward-mode AD and ``torch.func`` get the error that every custom function without a
rule for them gives.
"""
import torch

import _native as N


class Recorded(torch.autograd.Function):
    @staticmethod
    def forward(ctx, name, *args):
        state = torch._C._get_tracing_state()
        torch._C._set_tracing_state(None)                 # the op's own work is not part of the trace
        try:
            ins = [a.detach().requires_grad_(a.requires_grad) if isinstance(a, torch.Tensor) else a for a in args]
            with torch.enable_grad():
                out = getattr(N.ext(), name)(*ins)
            ctx.ins, ctx.outs = ins, out if isinstance(out, tuple) else (out,)
            outs = tuple(o.detach() for o in ctx.outs)
        finally:
            torch._C._set_tracing_state(state)
        if state is not None:
            outs = tuple(o.detach() for o in outs)        # a tracer has to have seen an op make each output
        return outs if isinstance(out, tuple) else outs[0]

    @staticmethod
    def backward(ctx, *grads):
        wrt = [a for a in ctx.ins if isinstance(a, torch.Tensor) and a.requires_grad]
        used = [(o, g) for o, g in zip(ctx.outs, grads) if g is not None and o.requires_grad]
        got = iter(torch.autograd.grad([o for o, _ in used], wrt, [g for _, g in used], retain_graph=True, allow_unused=True)
                   if used else [None] * len(wrt))
        return (None, *(next(got) if isinstance(a, torch.Tensor) and a.requires_grad else None for a in ctx.ins))
