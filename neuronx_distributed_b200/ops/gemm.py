"""bf16 GEMM on tcgen05 tensor cores (kernel: ``csrc/gemm_sm100.cu``).

``matmul(a, b, trans_a, trans_b)`` computes ``op(a) @ op(b)`` for row-major 2-D bf16 tensors with
fp32 accumulation in TMEM.  The three layouts training needs map to UMMA operand majors without
any transposition copies:

    fwd   : x[M,K] @ W[N,K]^T     → A K-major,  B K-major     ("nt")
    dgrad : g[M,K] @ W[K,N]       → A K-major,  B MN-major    ("nn")
    wgrad : g[K,M]^T @ x[K,N]     → A MN-major, B MN-major    ("tn")
"""
from __future__ import annotations

import os
from typing import Optional

import torch

from . import _ext

_MIN_DIM = 64
_USE_2CTA = os.environ.get("NXD_GEMM_2CTA", "1") == "1"   # CTA-pair kernel (cta_group::2)


def fused_wgrad_enabled() -> bool:
    return _ext.env("NXD_DISABLE_FUSED_WGRAD") != "1" and _ext.env("NXD_DISABLE_TCGEN05_GEMM") != "1"


def _eligible(a: torch.Tensor, b: torch.Tensor, M: int, N: int, K: int, any_rows: bool = False) -> bool:
    if _ext.env("NXD_DISABLE_TCGEN05_GEMM") == "1":
        return False
    if not (a.is_cuda and b.is_cuda and a.dtype == torch.bfloat16 and b.dtype == torch.bfloat16):
        return False
    if not (a.is_contiguous() and b.is_contiguous()) or a.data_ptr() % 16 or b.data_ptr() % 16:
        return False
    if not _ext.use_cuda(a, b) or not hasattr(_ext.ext(), "gemm_bf16"):
        return False
    # TMA needs 16-byte aligned rows; kernel handles ragged M/N/K tails via TMA zero fill
    return M >= 1 and N % 8 == 0 and K % 8 == 0 and (any_rows or M % 8 == 0)


def _few_rows(M: int, N: int, K: int) -> bool:
    """Rows for which streaming the weights decides the time (``csrc/gemm_few_sm100.cu``).  Up to 64 always (48 rows of 4096 x 11008:
    21 us against 69) and up to 128 unless the columns are so many that the wide tiles fill the GPU many times over (128 rows: 57344 x 8192
    168 against 171, 128256 x 4096 206 against 194).  Above, one block fits an SM, and it wins on long rows where the wide tiles would leave
    SMs idle (200 rows: 4096 x 11008 28 us against 71, 7168 x 8192 35 against 58; 9472 columns are 74 slabs of 128, one for each pair of
    SMs) or by its smaller padding (136 rows of 22016 x 4096: 57 against 65; 248: 73 against 68); on short rows it loses (176 rows:
    32000 x 512 29 against 26, 8192 x 1024 20 against 18)."""
    if M <= 128:
        return M <= 64 or N <= 65536
    return K >= 2048 and (N <= 9472 or (M <= 176 and N <= 65536)) and M < 256


def _pairs(M: int, N: int) -> bool:
    """Products for the CTA-pair kernel; the other one, tiles of 128 rows on single CTAs without a split of K, wins where at most 128 rows
    meet so many columns that its tiles fill the GPU (64 rows: 32000 x 4096 47 us against 56; but 128 rows of 4096 x 22016 129 against 43, of
    1024 x 5632 35 against 17, of 8192 x 7168 51 against 34).  The same line stands in ``csrc/native_autograd.cpp``."""
    return M > 128 or N <= 16384


def matmul(a: torch.Tensor, b: torch.Tensor, trans_a: bool = False, trans_b: bool = False,
           out: torch.Tensor | None = None, accumulate: bool = False, out_dtype=None) -> torch.Tensor:
    """``op(a) @ op(b)`` for 2-D tensors. ``accumulate`` adds into ``out`` (fp32 or bf16)."""
    M = a.shape[1] if trans_a else a.shape[0]
    K = a.shape[0] if trans_a else a.shape[1]
    N = b.shape[0] if trans_b else b.shape[1]
    out_dtype = out_dtype or (out.dtype if out is not None else a.dtype)
    if (M <= 8 and not trans_a and trans_b and out is None and out_dtype == torch.bfloat16 and a.is_cuda
            and a.dtype == torch.bfloat16 and b.dtype == torch.bfloat16 and K % 8 == 0 and a.is_contiguous() and b.is_contiguous()
            and _ext.ext() is not None and hasattr(_ext.ext(), "gemv") and _ext.env("NXD_DISABLE_TCGEN05_GEMM") != "1"):
        # decode-time GEMV: a bandwidth problem (every weight byte read once), not a tensor-core one — csrc/decode.cu
        _ext.count_launch()
        return _ext.ext().gemv(a, b, None)
    few = out is None and not trans_a and trans_b and out_dtype == torch.bfloat16 and _few_rows(M, N, K)
    # Rows that are no multiple of 8: cuBLAS, but for up to 64 rows of x·Wᵀ (9 / 33 / 49 rows of 11008 -> 4096: 17.7 / 19.3 / 20.3 us, 20.7 / 20.7 / 21.2;
    # 17 of 2816 -> 1024: 6.1 and 8.4; above, 97 of 3584 -> 8192: 17.6 and 14.9)
    if _eligible(a, b, M, N, K, few and M <= 64) and out_dtype in (torch.bfloat16, torch.float32):
        if out is not None and out.data_ptr() % 16:          # outputs leave through TMA or 16-byte stores: by way of a buffer
            res = matmul(a, b, trans_a, trans_b, out_dtype=torch.float32)
            return out.add_(res) if accumulate else out.copy_(res)
        if few:
            _ext.count_launch()
            return _ext.ext().gemm_few_rows(a, b)
        if out is None:
            out = torch.empty(M, N, dtype=out_dtype, device=a.device)
            accumulate = False
        _ext.count_launch()
        if _USE_2CTA and _pairs(M, N) and hasattr(_ext.ext(), "gemm_bf16_2cta"):
            _ext.ext().gemm_bf16_2cta(a, b, out, bool(trans_a), bool(trans_b), bool(accumulate))
        else:
            _ext.ext().gemm_bf16(a, b, out, bool(trans_a), bool(trans_b), bool(accumulate))
        return out
    if a.is_cuda and a.dtype == torch.bfloat16 and not _ext.env("NXD_DISABLE_TCGEN05_GEMM") \
            and (not a.is_contiguous() or not b.is_contiguous()):
        # make operands dense once and retry the tensor-core kernel
        return matmul(a.contiguous(), b.contiguous(), trans_a, trans_b, out, accumulate, out_dtype)
    aa = a.t() if trans_a else a
    bb = b.t() if trans_b else b
    res = torch.matmul(aa, bb)
    if out is not None:
        if accumulate:
            out.add_(res.to(out.dtype))
        else:
            out.copy_(res)
        return out
    return res.to(out_dtype)


def linear_swiglu(x: torch.Tensor, w: torch.Tensor, nodes=None) -> Optional[torch.Tensor]:
    """SwiGLU of ``x[..., K] @ w[2 I, K]^T`` (gate rows first) in one kernel, where there is one for it and it is faster than two: the
    few-row kernel up to 128 rows (48 rows of 4096 -> 2 x 11008: 36.9 us and 39.2, 9 of 1024 -> 2 x 2816: 5.8 and 7.3; above, where a block fills an
    SM, 129 rows 59.0 and 55.7), the CTA pairs from 136 rows on unless the few-row kernel takes them (1000 rows of 5120 -> 2 x 13824: the
    55 MB of products stay on the chip).  With gradients (``nodes``: those of ``_ext.native``) the CTA pairs alone."""
    K, N = x.shape[-1], w.shape[0]
    M = x.numel() // K if K else 0
    few = _few_rows(M, N, K)
    if w.dim() != 2 or (few and (M > 128 or (M > 64 and M % 8))):
        return None
    if nodes is not None:
        if (few or x.dim() < 2 or M % 8 or M <= 128 or N % 256 or K % 8 or not x.is_cuda or x.device != w.device or x.shape[-1] != w.shape[1]
                or not x.dtype == w.dtype == torch.bfloat16 or not x.is_contiguous() or not w.is_contiguous() or x.data_ptr() % 16 or w.data_ptr() % 16
                or M >= 2 ** 23):
            return None
        return nodes.linear_swiglu(x, w)
    y = _ext.ext().linear_swiglu(x, w, few)
    if y is not None:
        _ext.count_launch()
    return y


def linear_nt(x: torch.Tensor, w: torch.Tensor) -> torch.Tensor:
    """``x[..., K] @ w[N, K]^T``."""
    x2 = x.reshape(-1, x.shape[-1])
    return matmul(x2, w, False, True).view(*x.shape[:-1], w.shape[0])


# ---------------------------------------------------------------------------------------------------------------------
# Grouped (MoE blockwise) GEMM: rows of ``x`` come in ``block_size``-row blocks, block i is multiplied by the weights of
# expert ``block_to_expert[i]``.  CUDA: MODE 3 / 4 of ``csrc/gemm2cta_sm100.cu`` (the per-block expert only shifts the TMA
# coordinate of the weight tile — no per-block weight copies, no host sync); CPU / odd shapes: plain loop.
# Role of the reference's blockwise NKI kernels (modules/moe/blockwise.py:180-468, 1037-1127).
def _grouped_ok(x: torch.Tensor, w: torch.Tensor, block_size: int) -> bool:
    e = _ext.ext()
    return (x.is_cuda and e is not None and hasattr(e, "grouped_gemm") and x.dtype == torch.bfloat16
            and w.dtype == torch.bfloat16 and block_size % 128 == 0 and w.shape[1] % 64 == 0 and w.shape[2] % 64 == 0
            and _ext.env("NXD_DISABLE_GROUPED_GEMM") != "1")


def _grouped_ref(x, w, b2e, block_size):
    nb = b2e.numel()
    xb = x.view(nb, block_size, x.shape[-1])
    return torch.einsum("bth,bhi->bti", xb, w[b2e.long()]).reshape(nb * block_size, w.shape[-1])


class _GroupedMatmul(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, b2e, seg_first_block, block_size, skip_unused, slot_token):
        ctx.save_for_backward(x, w, b2e, seg_first_block, slot_token)
        ctx.block_size, ctx.skip_unused = block_size, skip_unused
        _ext.count_launch()
        return _ext.ext().grouped_gemm(x.contiguous(), w.contiguous(), b2e, block_size, False, seg_first_block if skip_unused else None)

    @staticmethod
    def backward(ctx, gy):
        x, w, b2e, seg, slot_token = ctx.saved_tensors
        return *_GroupedMatmul.gradients(ctx, gy, x, w, b2e, seg, slot_token), None, None, None, None, None

    @staticmethod
    def gradients(ctx, gy, x, w, b2e, seg, slot_token):
        extra = () if slot_token is None else (slot_token,)
        gy = gy.contiguous()
        gx = gw = None
        if ctx.needs_input_grad[0]:
            _ext.count_launch()
            gx = _ext.ext().grouped_gemm(gy, w.contiguous(), b2e, ctx.block_size, True, seg if ctx.skip_unused else None)       # dy · W[e]ᵀ
        if ctx.needs_input_grad[1]:
            _ext.count_launch()
            mg = getattr(w, "main_grad", None)
            if mg is not None and fused_wgrad_enabled() and mg.dtype == torch.float32 and mg.is_contiguous():
                fresh = getattr(w, "main_grad_fresh", False)
                _ext.ext().grouped_wgrad(x.contiguous(), gy, mg.view_as(w), seg, ctx.block_size, not fresh, *extra)
                w.main_grad_fresh = False
                cb = getattr(w, "_nxd_grad_ready", None)
                if cb is not None:
                    cb(w)
            else:
                gw = torch.empty_like(w)
                _ext.ext().grouped_wgrad(x.contiguous(), gy, gw, seg, ctx.block_size, False, *extra)
        return gx, gw


class _GroupedProducts(torch.autograd.Function):
    """``_GroupedMatmul`` over the used blocks, its ``products`` ([] around them: they are no input) computed already."""

    @staticmethod
    def forward(ctx, x, w, b2e, seg_first_block, block_size, slot_token, products):
        ctx.block_size, ctx.skip_unused = block_size, True
        ctx.save_for_backward(x, w, b2e, seg_first_block, slot_token)
        return products[0]

    @staticmethod
    def backward(ctx, gy):
        return *_GroupedMatmul.gradients(ctx, gy, *ctx.saved_tensors), None, None, None, None, None


def grouped_matmul(x: torch.Tensor, w: torch.Tensor, block_to_expert: torch.Tensor, seg_first_block: torch.Tensor,
                   block_size: int, skip_unused: bool = False, slot_token: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``y[i·B:(i+1)·B] = x[i·B:(i+1)·B] @ w[block_to_expert[i]]`` with ``x [nb·B, K]``, ``w [E, K, N]``.  With ``skip_unused``
    the row blocks from ``seg_first_block[E]`` on hold no tokens: their rows of the result are unspecified.  ``slot_token`` (int32 [nb·B], the
    token of each row): rows of -1 behind an expert's tokens are zero in ``x`` and in the gradient of ``y``, and the weight gradient skips them."""
    if _grouped_ok(x, w, block_size):
        return _GroupedMatmul.apply(x, w, block_to_expert.int(), seg_first_block.int(), block_size, skip_unused, slot_token)
    return _grouped_ref(x, w, block_to_expert, block_size)


def grouped_swiglu(x: torch.Tensor, w: torch.Tensor, block_to_expert: torch.Tensor, seg_first_block: torch.Tensor, block_size: int,
                   slot_token: Optional[torch.Tensor] = None) -> torch.Tensor:
    """SwiGLU of ``grouped_matmul(..., skip_unused=True)``.  Whole tiles of gates and ups on plain CUDA tensors that nobody records or traces: one
    kernel (8 experts, 4096 tokens of 2 choices, 4096 -> 2 x 3584, both ways, in turn: 1910 us and 2020; 1024 tokens 708 and 770)."""
    from . import act

    if (_grouped_ok(x, w, block_size) and block_size % 256 == 0 and w.shape[2] % 256 == 0 and x.shape[0] and x.device == w.device and x.dim() == 2
            and x.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0 and _ext.native(x, w) is not None):
        keep, b2e, seg = torch.is_grad_enabled() and (x.requires_grad or w.requires_grad), block_to_expert.int(), seg_first_block.int()
        _ext.count_launch()
        x = x.contiguous()
        with torch.no_grad():
            out = _ext.ext().grouped_swiglu(x, w.contiguous(), b2e, block_size, seg, keep)
        if not keep:
            return out[0]
        # two nodes: the products are given back before the gradients of rows and weights need memory
        return _ext.native(x, w).swiglu_of(_GroupedProducts.apply(x, w, b2e, seg, block_size, slot_token, out[1:]), out[0])
    return act.swiglu(grouped_matmul(x, w, block_to_expert, seg_first_block, block_size, skip_unused=True, slot_token=slot_token))
