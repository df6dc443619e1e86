"""Rotation out of the fused projection against the separate rotations."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,B,H,K,D", [(1, 1, 1, 1, 16), (37, 3, 6, 2, 128), (130, 1, 8, 8, 64), (5, 2, 40, 4, 128)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("strided", [False, True])
def test_rotary_qkv(S, B, H, K, D, dtype, strided):
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(S)
    x = torch.randn(S, B, (H + 2 * K) * D, generator=g, device="cuda").to(dtype).requires_grad_()
    cos, sin = ops.rope.rope_tables(S + 3, D, device="cuda")
    sections = x.split([H * D, K * D, K * D], -1)
    assert ops.rope.fused_qkv(*sections, cos, sin, H, K, D) is None
    sections[0]._qkv_sections = (x, *sections[1:])
    assert ops.rope.fused_qkv(sections[0], sections[1] * 1, sections[2], cos, sin, H, K, D) is None
    got = ops.rope.rotary_qkv(ops.rope.fused_qkv(*sections, cos, sin, H, K, D), cos, sin, H, K)
    q, k, v = (t.unflatten(-1, (-1, D)).transpose(0, 1) for t in x.split([H * D, K * D, K * D], -1))
    want = (ops.rope.apply_rotary(q, cos[:S], sin[:S]), ops.rope.apply_rotary(k, cos[:S], sin[:S]), v)
    grads = [torch.randn(B, S, h, D + 1 if strided else D, generator=g, device="cuda").to(dtype)[..., :D] for h in (H, K, K)]
    for a, b in zip(got, want):
        assert torch.equal(a, b) and a.stride() == b.stride()
    a, = torch.autograd.grad(got, x, grads)
    b, = torch.autograd.grad(want, x, grads)
    assert torch.equal(a, b)
