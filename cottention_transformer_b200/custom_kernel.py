"""Drop-in for ``Cuda_Kernel/Custom_Kernel.py``: the ``CustomAttention`` autograd Function.

Same contract as the reference (``Custom_Kernel.py:7-141``): ``forward(ctx, Q, K, V)`` makes the
inputs contiguous, saves them, and dispatches on ``Q.dtype`` to ``kernel.<dtype>(Q, K, V, 1, False,
False)`` (``:9-32``); ``backward`` runs the three permuted scans (``:106-108``)

    grad_Q = kernel(grad_output, V, K, rev=False)
    grad_K = kernel(V, grad_output, Q, rev=True)
    grad_V = kernel(K, Q, grad_output, rev=True)

each through the same name-dispatch, so the autocast rules of the entry points apply to the
backward exactly as they do in the reference.  Passes ``torch.autograd.gradcheck`` in float64, the
reference's only correctness check (``:184-188``), and ``gradgradcheck``: under ``create_graph`` the three
scans are differentiable themselves (the reference's kernel calls are not, and drop out of a second
derivative without a word).
"""
from __future__ import annotations

import torch

from . import _binding, kernel

_BY_DTYPE = {
    torch.float32: kernel.float32,
    torch.float64: kernel.float64,
    torch.float16: kernel.float16,
    torch.bfloat16: kernel.bfloat16,
}


def _scans(fn, g, Q, K, V, reversed):
    """The gradients of ``fn(Q, K, V, 1, False, reversed)``: three more scans."""
    return fn(g, V, K, 1, False, reversed), fn(V, g, Q, 1, False, not reversed), fn(K, Q, g, 1, False, not reversed)


class _Scan(torch.autograd.Function):
    """One scan in either direction through the entry point ``fn``, as often differentiable as one likes: its gradients are
    scans again."""

    @staticmethod
    def forward(ctx, Q, K, V, fn, reversed):
        ctx.save_for_backward(Q, K, V)
        ctx.fn, ctx.reversed = fn, reversed
        return fn(Q, K, V, 1, False, reversed)

    @staticmethod
    def backward(ctx, grad_output):
        return *_differentiable_scans(ctx.fn, grad_output.contiguous(), *ctx.saved_tensors, ctx.reversed), None, None


def _differentiable_scans(fn, g, Q, K, V, reversed):
    if not torch.is_grad_enabled():
        return _scans(fn, g, Q, K, V, reversed)
    return _scans(lambda q, k, v, _block, _inplace, rev: _Scan.apply(q, k, v, fn, rev), g, Q, K, V, reversed)


class CustomAttention(torch.autograd.Function):
    @classmethod
    def apply(cls, *args):
        """The same function with its autograd node in the compiled binding, where there is one to use."""
        if cls is CustomAttention and len(args) == 3 and all(isinstance(t, torch.Tensor) for t in args) and args[0].dtype in _BY_DTYPE:
            m = _binding.autograd()
            if m is not None:
                return m.custom_attention(*args)
            args = [t.contiguous() for t in args]  # (dense before the node: what it saves stays connected to the caller's tensors)
        return super().apply(*args)

    @staticmethod
    def forward(ctx, Q, K, V):
        Q = Q.contiguous()
        K = K.contiguous()
        V = V.contiguous()
        ctx.save_for_backward(Q, K, V)
        fn = _BY_DTYPE.get(Q.dtype)
        if fn is None:
            raise ValueError("Only float32, float64, float16, and bfloat16 are supported")
        return fn(Q, K, V, 1, False, False)

    @staticmethod
    def backward(ctx, grad_output):
        Q, K, V = ctx.saved_tensors
        Q = Q.contiguous()
        K = K.contiguous()
        V = V.contiguous()
        grad_output = grad_output.contiguous()
        fn = _BY_DTYPE.get(Q.dtype)
        if fn is None:
            raise ValueError("Only float32, float64, float16, and bfloat16 are supported")
        return _differentiable_scans(fn, grad_output, Q, K, V, False)
