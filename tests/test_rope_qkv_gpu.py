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


@pytest.mark.parametrize("watch", ["hook", "global hook", "wrapper", "own forward"])
def test_watched_projection_stays_in_the_graph(watch):
    """Whoever keeps q, k or v of the projection can ask for their gradients."""
    import torch.distributed as dist
    from torch.nn.modules.module import register_module_forward_hook

    from neuronx_distributed_b200 import ops
    from neuronx_distributed_b200.models.llama import LlamaAttention, LlamaConfig
    from neuronx_distributed_b200.parallel_layers import parallel_state as ps

    if not dist.is_initialized():
        dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1)
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(tensor_model_parallel_size=1)
    torch.manual_seed(0)
    att = LlamaAttention(LlamaConfig(hidden_size=256, num_attention_heads=2, num_key_value_heads=1, dtype=torch.bfloat16, device="cuda"))
    x = torch.randn(48, 2, 256, device="cuda").bfloat16().requires_grad_()
    go = torch.randn(48, 2, 256, device="cuda").bfloat16()
    cos, sin = ops.rope.rope_tables(48, 128, device="cuda")
    want, = torch.autograd.grad(att(x, cos, sin), x, go)
    proj, kept, handle = att.qkv_proj, [], None

    def keep(out):
        kept[:] = out
        return out

    if watch == "hook":
        proj.register_forward_hook(lambda m, i, o: (keep(o), None)[1])
    elif watch == "global hook":
        handle = register_module_forward_hook(lambda m, i, o: (keep(o), None)[1] if m is proj else None)
    elif watch == "wrapper":
        class Keep(torch.nn.Module):
            def __init__(self, inner):
                super().__init__()
                self.inner = inner

            def forward(self, t):
                return keep(self.inner(t))

        att.qkv_proj = Keep(proj)
    else:
        proj.forward = lambda t: keep(type(proj).forward(proj, t))
    try:
        y = att(x, cos, sin)
    finally:
        if handle is not None:
            handle.remove()
    *sections, got = torch.autograd.grad(y, (*kept, x), go)
    w = proj.weight_qkv.detach().double()
    back = torch.cat(sections, -1).double() @ w
    assert (got.double() - want.double()).norm() <= 2.0 ** -7 * want.double().norm()
    assert (got.double() - back).norm() <= 2.0 ** -7 * back.norm()      # one rounding to bfloat16 each
