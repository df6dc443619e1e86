"""Rows of routed experts in expert order (kernels: ``csrc/moe_blocks.cu``): slots, gather, weighted combine.

A :class:`Slots` holds where every (token, choice) of ``expert_index [T, k]`` goes when each expert's rows are padded to a
multiple of ``block`` rows; ``gather`` and ``combine`` move rows there and back and are each other's backward pass.
"""
from __future__ import annotations

from dataclasses import dataclass

import torch

from . import _ext

BLOCK = 256          # rows per block: one tile of the CTA-pair grouped GEMM


@dataclass
class Slots:
    expert_index: torch.Tensor     # [T, k] int64
    block_expert: torch.Tensor     # [nb] int32
    token: torch.Tensor            # [nb * block] int32, -1 = padding
    seg: torch.Tensor              # [E + 1] int32, first block of every expert; seg[E] = blocks that hold tokens
    slot: torch.Tensor             # [T * k] int32
    block: int


def usable(hidden: torch.Tensor, expert_index: torch.Tensor, num_experts: int) -> bool:
    e = _ext.ext() if hidden.is_cuda else None
    return (e is not None and hasattr(e, "moe_slots") and hidden.dtype == torch.bfloat16 and hidden.dim() == 2
            and hidden.shape[1] % 8 == 0 and num_experts <= 256 and expert_index.dim() == 2 and expert_index.numel() > 0)


def make_slots(expert_index: torch.Tensor, num_experts: int, num_blocks: int, block: int = BLOCK) -> Slots:
    idx = expert_index.long().contiguous()
    _ext.count_launch()
    b2e, token, seg, slot = _ext.ext().moe_slots(idx, int(num_experts), int(block), int(num_blocks))
    return Slots(idx, b2e, token, seg, slot, block)


def _rows(t: torch.Tensor) -> torch.Tensor:
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()      # the kernels move 16-byte packets


class _Gather(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, slots):
        ctx.slots = slots
        _ext.count_launch()
        return _ext.ext().moe_gather(_rows(x), slots.token, slots.seg, slots.block)

    @staticmethod
    def backward(ctx, g):
        s = ctx.slots
        _ext.count_launch()
        return _ext.ext().moe_combine(_rows(g), s.slot, s.expert_index, None), None


class _Combine(torch.autograd.Function):
    @staticmethod
    def forward(ctx, y, weight, slots):
        ctx.slots = slots
        y, weight = _rows(y), weight.contiguous()
        ctx.save_for_backward(y, weight)
        _ext.count_launch()
        return _ext.ext().moe_combine(y, slots.slot, slots.expert_index, weight)

    @staticmethod
    def backward(ctx, g):
        (y, weight), s = ctx.saved_tensors, ctx.slots
        _ext.count_launch()
        dy, dw = _ext.ext().moe_combine_grad(_rows(g), y, s.token, s.block_expert, s.seg, weight, s.block)
        return dy, dw, None


class _Normalize(torch.autograd.Function):
    @staticmethod
    def forward(ctx, aff, idx):
        ctx.save_for_backward(aff, idx)
        _ext.count_launch()
        return _ext.ext().moe_normalize(aff.contiguous(), idx)

    @staticmethod
    def backward(ctx, g):
        aff, idx = ctx.saved_tensors
        if torch.is_grad_enabled():                         # create_graph: the gradient is differentiated again
            mask = torch.zeros_like(aff).scatter_(1, idx, 1.0)
            a = aff * mask
            total = a.sum(-1, keepdim=True)
            s = total.clamp(min=1e-9)
            return (g / s - (g * a / s / s).sum(-1, keepdim=True) * (total >= 1e-9)) * mask, None
        _ext.count_launch()
        return _ext.ext().moe_normalize_grad(g.contiguous(), aff.contiguous(), idx), None


def normalize_ok(aff: torch.Tensor, expert_index: torch.Tensor) -> bool:
    """fp32 ``[T, E]`` on the device with int64 choices, in a call that nobody records, traces or transforms."""
    return (aff.dtype == torch.float32 and aff.dim() == 2 and aff.shape[1] <= 256 and expert_index.dtype == torch.int64 and expert_index.dim() == 2
            and expert_index.device == aff.device and expert_index.shape[0] == aff.shape[0] and _ext.native(aff, expert_index) is not None)


def normalize(aff: torch.Tensor, expert_index: torch.Tensor) -> torch.Tensor:
    """Affinities ``[T, E]`` of the chosen experts divided by their sum (at least 1e-9); the others zero."""
    return _Normalize.apply(aff, expert_index.contiguous())


def gather(x: torch.Tensor, slots: Slots) -> torch.Tensor:
    """``x [T, H]`` → rows in slot order ``[nb * block, H]``; padding rows are zero, rows behind the last used block unspecified."""
    return _Gather.apply(x, slots)


def combine(y: torch.Tensor, weight: torch.Tensor, slots: Slots) -> torch.Tensor:
    """``out[t] = sum_j weight[t, e_j] * y[slot(t, j)]`` with fp32 ``weight [T, E]`` and fp32 sums."""
    return _Combine.apply(y, weight, slots)
