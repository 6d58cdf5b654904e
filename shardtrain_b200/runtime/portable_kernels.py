"""Autograd nodes of the portable executor that run as one kernel each on a GPU (`csrc/portable.cu`).

They compute what `models.qwen2.apply_rotary` + `causal_attention` and `swiglu` compute, with the same
roundings; `usable` says whether a call can be served, otherwise the caller keeps the torch operators (CPU,
other dtypes, autocast, 4-D masks).
"""

from __future__ import annotations

import torch
from torch.autograd.function import once_differentiable

from shardtrain_b200 import ops as ops_module

_DTYPES = (torch.float32, torch.float16, torch.bfloat16)


def usable(*tensors) -> bool:
    first = tensors[0]
    return (first.is_cuda and first.dtype in _DTYPES and not torch.is_autocast_enabled("cuda")
            and all(t.is_cuda and t.dtype == first.dtype for t in tensors)
            and ops_module.extension_path() is not None)


class Attention(torch.autograd.Function):
    """Rotary positions and grouped-query causal attention on the projections' outputs.

    q [B, S, hq * d], k and v [B, S, hkv * d], cos and sin fp32 [1 or B, S, d], mask None or [B, S] ->
    [B, S, hq * d].  The query heads of a group are stacked along the rows of one product per key head, so
    k and v are not repeated.  Saved: the rotated operands, the scores as the product left them and the rows'
    maximum and sum; the backward forms the fp32 probabilities again.
    """

    @staticmethod
    def forward(ctx, q, k, v, cos, sin, mask, d):
        ops = ops_module.load()
        batch, seq, width = q.shape
        qr, kr, vr = ops.portable_rotate(q, k, v, cos, sin, d)
        kv_heads = kr.shape[1]
        grouped = qr.view(batch, kv_heads, -1, d)
        scores = torch.matmul(grouped, kr.transpose(-1, -2))
        probs, stats = ops.portable_softmax(scores, mask, d)
        out = torch.matmul(probs, vr).view(batch, -1, seq, d)
        ctx.save_for_backward(grouped, kr, vr, scores, probs, stats, cos, sin, mask)
        ctx.d = d
        return out.transpose(1, 2).reshape(batch, seq, width)

    @staticmethod
    @once_differentiable
    def backward(ctx, grad):
        ops = ops_module.load()
        grouped, kr, vr, scores, probs, stats, cos, sin, mask = ctx.saved_tensors
        d = ctx.d
        batch, kv_heads, seq, _ = kr.shape
        g = grad.reshape(batch, seq, -1, d).transpose(1, 2).reshape(batch, kv_heads, -1, d)

        def over_queries(left, right):
            """left^T right summed over the queries and heads of each group: in 16 bits by one product (one
            rounding); in fp32 head by head, as one sum over all of them is twice as far from exact."""
            if left.dtype != torch.float32 or left.shape[2] == seq:
                return torch.matmul(left.transpose(-1, -2), right)
            left, right = (t.view(batch, kv_heads, -1, seq, t.shape[-1]) for t in (left, right))
            return torch.matmul(left.transpose(-1, -2), right).sum(2)

        dv = over_queries(probs, g)
        ds = ops.portable_softmax_bwd(scores, mask, stats, torch.matmul(g, vr.transpose(-1, -2)), d)
        dq = torch.matmul(ds, kr).view(batch, -1, seq, d)
        dk = over_queries(ds, grouped)
        return (*ops.portable_rotate_bwd(dq, dk, dv, cos, sin), None, None, None, None)


def attention(q, k, v, tables, attention_mask, d):
    """`Attention` where it can serve the call, else None."""
    cos, sin = tables
    if not (usable(q, k, v) and cos.is_cuda and cos.dtype == sin.dtype == torch.float32 and d % 2 == 0
            and cos.ndim == 3 and cos.shape[0] in (1, q.shape[0]) and cos.shape[1:] == (q.shape[1], d)
            and q.numel()):
        return None
    mask = None
    if attention_mask is not None:
        if attention_mask.shape != q.shape[:2]:
            return None                       # 4-D forms; a wrong shape is refused there too
        mask = attention_mask.to(q.device).ne(0).contiguous()
    return Attention.apply(q.contiguous(), k.contiguous(), v.contiguous(), cos.contiguous(),
                           sin.contiguous(), mask, d)


class SwiGLU(torch.autograd.Function):
    @staticmethod
    def forward(ctx, gate, up):
        ctx.save_for_backward(gate, up)
        return ops_module.load().portable_swiglu(gate, up)

    @staticmethod
    @once_differentiable
    def backward(ctx, grad):
        gate, up = ctx.saved_tensors
        return ops_module.load().portable_swiglu_bwd(grad.contiguous(), gate, up)


def swiglu(gate, up):
    """`SwiGLU` where it can serve the call, else None."""
    if not usable(gate, up) or gate.shape != up.shape:
        return None
    return SwiGLU.apply(gate.contiguous(), up.contiguous())
