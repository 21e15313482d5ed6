"""DSA sparse attention (reference src/kernels.py:913-1312) on the hand-written kernels.

``sparse_attention(q, k, v, idx, scale=None)`` and ``SparseAttentionFunction`` keep the reference's names,
argument order, return values and dtypes: ``(output [B, H, L, D_v] in the inputs' dtype, attn_weights
[B, H, L, K] fp32)``, gradients for q, k, v in the inputs' dtype.  Both directions are one native
call (csrc/host/attention.cpp); ``sparse_attention`` is a native autograd node around them.
"""
from __future__ import annotations

import torch

from . import _lib

_host = _lib.host
_TAG = {torch.bfloat16: _lib.BF16, torch.float32: _lib.F32, torch.float16: _lib.F16}


class SparseAttentionFunction(torch.autograd.Function):
    """Autograd function with the reference's signature (src/kernels.py:1189-1289)."""

    @staticmethod
    def forward(ctx, q, k, v, idx, scale):
        out, attn, *saved = _host.attention_forward(q, k, v, idx, float(scale))
        ctx.save_for_backward(*saved)
        ctx.scale = float(scale)
        ctx.in_dtype = q.dtype
        ctx.mark_non_differentiable(attn)
        return out, attn

    @staticmethod
    def backward(ctx, grad_output, grad_attn_weights):
        return (*_host.attention_backward(grad_output, *ctx.saved_tensors, ctx.scale, torch.empty(0, dtype=ctx.in_dtype)), None, None)


def sparse_attention(q, k, v, idx, scale=None):
    """Attention over the K selected positions of every query (reference src/kernels.py:1292-1312).
    q, k: [B, H, L, D_qk]; v: [B, H, L, D_v]; idx: [B, L, K] int64.  Returns ``(output, attn_weights)``."""
    if scale is None:
        scale = q.shape[-1] ** -0.5
    return _host.attention(q, k, v, idx, scale)
