"""Routed experts on the block kernels against plain PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _experts(E, H, I):
    import torch.distributed as dist

    from neuronx_distributed_b200.modules.moe import ExpertMLPsV2, RoutedExpertsMLPOpsConfig
    from neuronx_distributed_b200.parallel_layers import parallel_state as ps

    if not dist.is_initialized():
        dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1)
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(tensor_model_parallel_size=1)
    cfg = RoutedExpertsMLPOpsConfig(num_experts=E, top_k=2, hidden_size=H, intermediate_size=I, hidden_act="silu", glu_mlp=True,
                                    capacity_factor=None, normalize_top_k_affinities=False)
    return ExpertMLPsV2(cfg, dtype=torch.bfloat16, device="cuda").train()


def _reference(x, aff, idx, w1, w2):
    out = torch.zeros_like(x)
    for j in range(idx.shape[1]):
        for e in range(w1.shape[0]):
            rows = (idx[:, j] == e).nonzero().squeeze(1)
            gate, up = (x[rows] @ w1[e]).chunk(2, -1)
            out = out.index_add(0, rows, (torch.nn.functional.silu(gate) * up) @ w2[e] * aff[rows, e].unsqueeze(1))
    return out


@pytest.mark.parametrize("T,E,H,I,choice", [(37, 8, 256, 192, "random"), (512, 4, 128, 64, "one expert"), (1025, 3, 320, 128, "random"),
                                            (700, 16, 128, 128, "twice"), (3000, 130, 64, 64, "random")])
def test_experts(T, E, H, I, choice):
    from neuronx_distributed_b200.modules.moe import blockwise

    m = _experts(E, H, I)
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, H, generator=g, device="cuda").bfloat16().requires_grad_()
    aff = torch.rand(T, E, generator=g, device="cuda").requires_grad_()
    idx = torch.stack([torch.randperm(E, generator=g, device="cuda")[:2] for _ in range(T)])
    if choice == "one expert":                              # the others get no tokens: zero weight gradients
        idx[:] = torch.tensor([1, 2], device="cuda")
    if choice == "twice":
        idx[:, 1] = idx[:, 0]
    w1, w2 = m.mlp_op.gate_up_proj.weight, m.mlp_op.down_proj.weight
    with torch.no_grad():
        for w in (w1, w2):
            w.copy_(torch.randn(w.shape, generator=g, device="cuda") * w.shape[1] ** -0.5)
    go = torch.randn(T, H, generator=g, device="cuda").bfloat16()
    assert blockwise._grouped_swiglu_ok(x, idx, m.mlp_op, E)
    y = blockwise.blockwise_expert_mlp(x, aff, idx, m.mlp_op, 512)
    got = [y, *torch.autograd.grad(y, (x, aff, w1, w2), go)]
    ref = [t.detach().double().requires_grad_() for t in (x, aff, w1, w2)]
    z = _reference(ref[0], ref[1], idx, ref[2], ref[3])
    want = [z, *torch.autograd.grad(z, ref, go.double())]
    # inputs of every product are rounded to bfloat16 once (2^-9), two to three in a row on each path
    for a, b in zip(got, want):
        assert (a.double() - b).norm() <= 0.012 * b.norm()
    for e in range(E):
        if not (idx == e).any():
            assert not got[3][e].any() and not got[4][e].any()


@pytest.mark.parametrize("T,E,H,I", [(40, 4, 64, 128), (700, 8, 320, 256), (1500, 3, 1024, 1408)])
@pytest.mark.parametrize("grads", [False, True])
def test_gated_products_are_those_of_two_kernels(T, E, H, I, grads):
    """The same tiles and sums, SwiGLU of the same rounded products: the same bits, in the rows of blocks with tokens, both ways."""
    from neuronx_distributed_b200 import ops

    mb = ops.moe_blocks
    g = torch.Generator(device="cuda").manual_seed(T)
    idx = torch.stack([torch.randperm(E, generator=g, device="cuda")[:2] for _ in range(T)])
    slots = mb.make_slots(idx, E, (2 * T + mb.BLOCK - 1) // mb.BLOCK + E)
    hidden = torch.randn(T, H, generator=g, device="cuda").bfloat16()
    w = (torch.randn(E, H, 2 * I, generator=g, device="cuda") * H ** -0.5).bfloat16().requires_grad_(grads)
    x = mb.gather(hidden, slots).detach().requires_grad_(grads)
    before = ops._ext.launches()
    one = ops.gemm.grouped_swiglu(x, w, slots.block_expert, slots.seg, mb.BLOCK, slots.token)
    assert ops._ext.launches() - before == 1
    two = ops.act.swiglu(ops.gemm.grouped_matmul(x, w, slots.block_expert, slots.seg, mb.BLOCK, skip_unused=True, slot_token=slots.token))
    used = int(slots.seg[-1]) * mb.BLOCK
    assert torch.equal(one[:used], two[:used]) and one.requires_grad == grads
    if grads:
        go = torch.randn_like(one) * (slots.token >= 0).unsqueeze(1)
        a, b = (torch.autograd.grad(y, (x, w), go) for y in (one, two))
        assert torch.equal(a[0][:used], b[0][:used]) and torch.equal(a[1], b[1])


@pytest.mark.parametrize("n,E,block", [(1, 1, 128), (1023, 5, 256), (1025, 256, 128), (70000, 33, 256)])
def test_slots(n, E, block):
    from neuronx_distributed_b200 import ops
    from neuronx_distributed_b200.modules.moe.blockwise import build_block_metadata, get_num_blocks

    g = torch.Generator(device="cuda").manual_seed(n)
    idx = torch.randint(0, E, (n, 1), generator=g, device="cuda")
    s = ops.moe_blocks.make_slots(idx, E, get_num_blocks(n, 1, E, block), block)
    b2e, tp2id, counts = build_block_metadata(idx.cpu(), E, block)
    assert torch.equal(s.token.cpu().long(), tp2id) and torch.equal(s.block_expert.cpu().long(), b2e)
    assert torch.equal(s.token[s.slot.long()].cpu().long(), torch.arange(n))
    first = torch.cat([torch.zeros(1, dtype=torch.long), torch.cumsum((counts + block - 1) // block, 0)])
    assert torch.equal(s.seg.cpu().long(), first)
    for a, b in zip(build_block_metadata(idx, E, block), (b2e, tp2id, counts)):
        assert torch.equal(a.cpu(), b)


def test_experts_with_an_activation_of_their_own():
    from neuronx_distributed_b200.modules.moe import blockwise

    m = _experts(4, 128, 64)
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(200, 128, generator=g, device="cuda").bfloat16()
    aff, idx = torch.rand(200, 4, generator=g, device="cuda"), torch.randint(0, 4, (200, 1), generator=g, device="cuda")
    op = m.mlp_op
    want = blockwise.blockwise_expert_mlp(x, aff, idx, op, 128)
    plain = type(op)
    op.activation = lambda h: 2 * plain.activation(op, h)                 # on the object
    assert not blockwise._grouped_swiglu_ok(x, idx, op, 4)
    got = [blockwise.blockwise_expert_mlp(x, aff, idx, op, 128)]
    del op.activation
    op.__class__ = type("Doubled", (plain,), {"activation": lambda self, h: 2 * plain.activation(self, h)})      # of its class
    assert not blockwise._grouped_swiglu_ok(x, idx, op, 4)
    got.append(blockwise.blockwise_expert_mlp(x, aff, idx, op, 128))
    for y in got:                                           # roundings to bfloat16 on the way, as in test_experts
        assert (y.double() - 2 * want.double()).norm() <= 0.012 * 2 * want.double().norm()


@pytest.mark.parametrize("T,E,k,scale", [(1, 1, 1, 1.0), (5, 8, 2, 1.0), (700, 33, 4, 1.0), (129, 256, 8, 1.0), (9, 256, 40, 1.0), (64, 16, 2, 1e-11)])
def test_normalized_affinities(T, E, k, scale):
    """Against the chain of plain operations in 64 bits; an expert chosen twice counts once, sums below 1e-9 count as 1e-9."""
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(T + E)
    aff = (torch.rand(T, E, generator=g, device="cuda") * scale).requires_grad_()
    idx = torch.randint(0, E, (T, k), generator=g, device="cuda")
    go = torch.randn(T, E, generator=g, device="cuda")
    assert ops.moe_blocks.normalize_ok(aff, idx)
    w = ops.moe_blocks.normalize(aff, idx)
    got = [w, *torch.autograd.grad(w, aff, go)]
    a = aff.detach().double().requires_grad_()
    m = a * torch.zeros_like(a).scatter_(1, idx, 1.0)
    z = m / m.sum(-1, keepdim=True).clamp(min=1e-9)
    # sums of up to 256 products in 32 bits, then two quotients: 1e-5 of w, and of what the gradient (go - sum of go * w) / sum subtracts: with
    # one expert it is zero, a difference of two numbers of the size of go / sum
    size = (go.double().abs().amax(-1) / m.detach().sum(-1).clamp(min=1e-9)).max()
    for x, y, bound in zip(got, [z, *torch.autograd.grad(z, a, go.double())], (1.0, size)):
        assert (x.double() - y).abs().max() <= 1e-5 * bound


def test_normalized_affinities_that_are_no_numbers():
    from neuronx_distributed_b200 import ops

    aff = torch.rand(4, 8, device="cuda")
    aff[0, 3], aff[1, 2], aff[2, 5] = float("nan"), float("inf"), float("nan")
    idx = torch.tensor([[3, 1], [2, 0], [0, 1], [6, 7]], device="cuda")
    mask = torch.zeros_like(aff).scatter_(1, idx, 1.0)
    want = aff * mask
    want = want / want.sum(-1, keepdim=True).clamp(min=1e-9)
    torch.testing.assert_close(ops.moe_blocks.normalize(aff, idx), want, equal_nan=True, rtol=1e-6, atol=0)


@pytest.mark.parametrize("counts", [[0, 1, 63, 64, 65], [255, 0, 256, 257, 128], [0, 0, 0, 0, 7], [320, 129, 191, 192, 193]])
@pytest.mark.parametrize("accumulate", [False, True])
def test_weight_gradients_without_padding(counts, accumulate):
    """Rows behind an expert's tokens are zero, so that leaving their k-blocks out changes no bit."""
    from neuronx_distributed_b200 import ops

    E, H, I, block = len(counts), 320, 192, 256
    idx = torch.cat([torch.full((n,), e) for e, n in enumerate(counts)])[:, None].cuda()
    nb = sum((n + block - 1) // block for n in counts) + 1
    s = ops.moe_blocks.make_slots(idx, E, nb, block)
    g = torch.Generator(device="cuda").manual_seed(sum(counts))
    x, dy = (torch.randn(nb * block, n, generator=g, device="cuda").bfloat16() * (s.token >= 0)[:, None] for n in (H, I))
    out = [torch.full((E, H, I), 0.5 if accumulate else float("nan"), device="cuda") for _ in range(2)]
    ops._ext.ext().grouped_wgrad(x, dy, out[0], s.seg, block, accumulate)
    ops._ext.ext().grouped_wgrad(x, dy, out[1], s.seg, block, accumulate, s.token)
    assert torch.equal(out[0], out[1]) and torch.isfinite(out[1]).all()


@pytest.mark.parametrize("strided", [False, True])
def test_normalized_affinities_are_differentiated_twice(strided):
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(5)
    T, E = 90, 12
    leaf = torch.rand((E, T) if strided else (T, E), generator=g, device="cuda").requires_grad_()
    idx = torch.randint(0, E, (T, 3), generator=g, device="cuda")
    go = torch.randn(T, E, generator=g, device="cuda")
    results = []
    for kernel in (True, False):
        aff = leaf.double() if not kernel else leaf
        aff = aff.t() if strided else aff
        assert not kernel or ops.moe_blocks.normalize_ok(aff, idx)
        m = aff * torch.zeros_like(aff).scatter_(1, idx, 1.0)
        w = ops.moe_blocks.normalize(aff, idx) if kernel else m / m.sum(-1, keepdim=True).clamp(min=1e-9)
        (first,) = torch.autograd.grad((w.square() * go).sum(), leaf, create_graph=True)
        results.append([first, *torch.autograd.grad(first.square().sum(), leaf)])
    for a, b in zip(*results):                # sums of up to three products and quotients in 32 bits, twice
        assert (a.double() - b).norm() <= 1e-5 * b.norm()
