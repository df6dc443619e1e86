"""Rotary position embedding, HF "rotate-half" convention, applied in place to q and k
(kernel: ``csrc/elementwise.cu`` rope_apply).  Backward is the same rotation with −sin.
Reference: ``overrides/transformer_overrides.py:20-32``, ``modules/attention/utils.py:50-80``.

Layout: q/k ``[B, S, H, D]`` (any strides on B/S/H as long as D is contiguous); cos/sin ``[S, D/2]``
fp32 (position ``s`` of the *global* sequence; callers slice for CP/SP offsets).
"""
from __future__ import annotations

import torch

from . import _ext


def _rope_ref(x, cos, sin, sign):
    # x [B,S,H,D]; cos/sin [S, D/2]
    d2 = x.shape[-1] // 2
    xf = x.float()
    x1, x2 = xf[..., :d2], xf[..., d2:]
    c = cos[None, :, None, :].float()
    s = sin[None, :, None, :].float() * sign
    return torch.cat([x1 * c - x2 * s, x2 * c + x1 * s], dim=-1).to(x.dtype)


class _Rope(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, cos, sin):
        ctx.save_for_backward(cos, sin)
        if _ext.use_cuda(x, cos, sin) and x.dtype in (torch.bfloat16, torch.float16, torch.float32) \
                and x.stride(-1) == 1 and x.shape[-1] % 2 == 0:
            ctx.cuda = True
            _ext.count_launch()
            return _ext.ext().rope_apply(x, cos.contiguous().float(), sin.contiguous().float(), 1.0)
        ctx.cuda = False
        return _rope_ref(x, cos, sin, 1.0)

    @staticmethod
    def backward(ctx, g):
        cos, sin = ctx.saved_tensors
        if ctx.cuda:
            _ext.count_launch()
            return _ext.ext().rope_apply(g, cos.contiguous().float(), sin.contiguous().float(), -1.0), None, None
        return _rope_ref(g, cos, sin, -1.0), None, None


def apply_rotary(x: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor) -> torch.Tensor:
    return _Rope.apply(x, cos, sin)


class _RopeQKV(torch.autograd.Function):
    """Rotated q and k and the view v of a fused projection output; backward fills ONE fused gradient (no concatenation)."""

    @staticmethod
    def forward(ctx, qkv, cos, sin, heads, kv_heads):
        cos, sin = cos.contiguous().float(), sin.contiguous().float()
        ctx.save_for_backward(cos, sin)
        _ext.count_launch()
        q, k = _ext.ext().rope_qkv_fwd(qkv, cos, sin, int(heads), int(kv_heads))
        D = q.shape[-1]
        v = qkv[..., (heads + kv_heads) * D:].unflatten(-1, (kv_heads, D))
        return q, k, v.transpose(0, 1)

    @staticmethod
    def backward(ctx, gq, gk, gv):
        cos, sin = ctx.saved_tensors
        _ext.count_launch()
        return _ext.ext().rope_qkv_bwd(_packets(gq), _packets(gk), _packets(gv), cos, sin), None, None, None, None


def _packets(t: torch.Tensor) -> torch.Tensor:
    per = 16 // t.element_size()
    ok = t.stride(3) == 1 and t.data_ptr() % 16 == 0 and all(t.shape[d] == 1 or t.stride(d) % per == 0 for d in range(3))
    return t if ok else t.contiguous()


def fused_qkv(q, k, v, cos, sin, heads: int, kv_heads: int, head_dim: int):
    """The projection output ``[S, B, (heads + 2 kv_heads) head_dim]`` whose sections ``q``, ``k`` and ``v`` still are, when
    :func:`rotary_qkv` takes it (whole 16-byte packets in each half of a head); None when one of the three was replaced on the way
    (an adapter) or carries a hook, or the sizes are for the separate rotations.  The sections leave the autograd graph: the caller
    makes sure that nobody else holds one."""
    sections = getattr(q, "_qkv_sections", None)
    if not isinstance(sections, tuple) or sections[1] is not k or sections[2] is not v:
        return None
    qkv = sections[0]
    if any(t._backward_hooks or t.retains_grad for t in (q, k, v)):
        return None
    if (qkv.dim() != 3 or qkv.dtype not in (torch.bfloat16, torch.float16, torch.float32) or head_dim % 2
            or qkv.shape[-1] != (heads + 2 * kv_heads) * head_dim or (head_dim // 2 * qkv.element_size()) % 16
            or not qkv.is_contiguous() or qkv.data_ptr() % 16 or cos.dim() != 2 or cos.shape != sin.shape
            or cos.shape[0] < qkv.shape[0] or cos.shape[1] != head_dim // 2 or not _ext.use_cuda(qkv, cos, sin)):
        return None
    return qkv


def rotary_qkv(qkv: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, heads: int, kv_heads: int):
    """``qkv [S, B, (heads + 2 kv_heads) D]`` → rotated ``q [B, S, heads, D]``, ``k`` and the view ``v [B, S, kv_heads, D]``:
    :func:`apply_rotary` of the first two sections, each direction one launch (``csrc/elementwise.cu`` rope_qkv)."""
    n = _ext.native(qkv, cos, sin)
    if n is not None:
        return n.rope_qkv(qkv, cos, sin, heads, kv_heads)
    return _RopeQKV.apply(qkv, cos, sin, heads, kv_heads)


def rope_tables(seq_len: int, dim: int, base: float = 10000.0, device=None, offset: int = 0,
                scaling: float = 1.0):
    inv = 1.0 / (base ** (torch.arange(0, dim, 2, dtype=torch.float32, device=device) / dim))
    t = (torch.arange(offset, offset + seq_len, dtype=torch.float32, device=device)) / scaling
    fr = torch.outer(t, inv)
    return fr.cos(), fr.sin()
