"""Calls recorded by torch.jit.trace.

The native operations (csrc/torch/ops.cpp) launch their kernels on raw pointers: a tracer sees the
allocation of the result and nothing else, and a replay would return that memory as it is.  While a
trace is being recorded, a call therefore goes through a Python autograd function, which the
tracer records as one operation and replays on its new inputs, gradients included.  (A call that
works in place cannot be replayed by the interpreter; the softmax refuses to be recorded.)
"""
import torch

recording = torch._C._get_tracing_state     # None unless a trace is being recorded


class _Recorded(torch.autograd.Function):

    @staticmethod
    def forward(ctx, op, method, *args):
        """`args`: tensors and plain values, as `op`'s method takes them.  The same `op` has to come
        again when the call is traced again: the tracer compares the two recordings."""
        grads = ctx.needs_input_grad[2:]
        args = tuple(x.detach().requires_grad_(g) if isinstance(x, torch.Tensor) else x for x, g in zip(args, grads))
        with torch.set_grad_enabled(any(grads)):
            out = getattr(op, method)(*args)
        ctx.inner = [x if g else None for x, g in zip(args, grads)], out
        return out.detach()

    @staticmethod
    def backward(ctx, grad):
        leaves, out = ctx.inner
        got = iter(torch.autograd.grad(out, [x for x in leaves if x is not None], grad, retain_graph=True, allow_unused=True))
        return (None, None) + tuple(None if x is None else next(got) for x in leaves)


def call(op, method, *args):
    return _Recorded.apply(op, method, *args)
