"""Backward attention whose K/V heads are shared by several blocks: fp32 sums of the parts against one block per K/V head."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,S,H,Hkv", [(1, 1, 2, 1), (2, 127, 6, 2), (1, 129, 8, 1), (1, 300, 16, 4)])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("sbhd", [True, False])
def test_parts_of_a_group(B, S, H, Hkv, causal, sbhd):
    from neuronx_distributed_b200.ops import _ext

    ext = _ext.ext()
    g = torch.Generator(device="cuda").manual_seed(S)
    q, k, v, go = (torch.randn(B, S, h, 128, generator=g, device="cuda").bfloat16() for h in (H, Hkv, Hkv, H))
    scale = 128 ** -0.5
    o, lse = ext.flash_attn_fwd(q, k, v, causal, scale, sbhd)
    want = ext.flash_attn_bwd(go, q, k, v, o, lse, causal, scale, sbhd, parts=1)
    qf, kf, vf = (t.double().transpose(1, 2).requires_grad_() for t in (q, k, v))
    s = qf @ kf.repeat_interleave(H // Hkv, 1).transpose(-1, -2) * scale
    if causal:
        s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    ref = torch.autograd.grad(s.softmax(-1) @ vf.repeat_interleave(H // Hkv, 1), (qf, kf, vf), go.double().transpose(1, 2))
    for parts in [p for p in range(2, H // Hkv + 1) if H // Hkv % p == 0] + [0]:
        got = ext.flash_attn_bwd(go, q, k, v, o, lse, causal, scale, sbhd, parts=parts)
        for a, b, r in zip(got, want, ref):
            assert a.stride() == b.stride()
            r = r.transpose(1, 2)
            # the same products in fp32, added in another order: a bf16 result moves by at most one step where it lies near a midpoint
            assert ((a.float() - b.float()).abs() <= 2 ** -7 * b.float().abs() + 1e-5 * b.float().abs().max()).all()
            assert (a.double() - r).norm() <= 1.05 * (b.double() - r).norm() + 1e-12
    with pytest.raises(RuntimeError):
        ext.flash_attn_bwd(go, q, k, v, o, lse, causal, scale, sbhd, parts=H // Hkv * 2)
