"""Kernels of the training step at the edges of their chunks: optimizer tables, embedding gradients, vocabulary loss."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _groups():
    import torch.distributed as dist

    from neuronx_distributed_b200.parallel_layers import parallel_state as ps

    if not dist.is_initialized():
        dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1)
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(tensor_model_parallel_size=1)


@pytest.mark.parametrize("sizes", [[1, 3, 0, 8191], [8192, 8193, 5], [7] * 60 + [40000], [3000000]])
@pytest.mark.parametrize("gdtype", [torch.float32, torch.bfloat16])
def test_optimizer_tables(sizes, gdtype):
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(len(sizes))
    p, m, v = ([torch.rand(n, generator=g, device="cuda") for n in sizes] for _ in range(3))
    gr = [torch.randn(n, generator=g, device="cuda").to(gdtype) for n in sizes]
    low = [t.bfloat16() for t in p]
    want = []
    scale, lr, b1, b2, eps, wd, step = 0.5, 1e-2, 0.9, 0.99, 1e-6, 0.1, 3
    for a, b, c, d in zip(p, gr, m, v):
        gg, a, c, d = (t.double() for t in (b, a, c, d))
        gg = gg * scale
        c, d = b1 * c + (1 - b1) * gg, b2 * d + (1 - b2) * gg * gg
        a = a - lr * math.sqrt(1 - b2 ** step) / (1 - b1 ** step) * c / (d.sqrt() + eps)
        want.append((a * (1 - lr * wd), c, d))
    total = sum(float((t.double() ** 2).sum()) for t in gr)
    # fp32 sums in chunks of 4096 elements and one atomic per block
    assert abs(float(ops.optim.multi_tensor_sq_norm(gr)) - total) <= 2.0 ** -19 * max(total, 1e-9)
    ops.optim.fused_adamw_(p, gr, m, v, lr, b1, b2, eps, wd, step, torch.tensor(scale, device="cuda"), low)
    for i, w in enumerate(want):
        for a, b in zip((p[i], m[i], v[i]), w):
            if a.numel():
                assert ((a.double() - b).abs() <= 2.0 ** -18 * (1 + b.abs())).all()
        assert torch.equal(low[i], p[i].bfloat16())
    before = [t.clone() for t in gr]
    ops.optim.multi_tensor_scale_(gr, 0.25)
    assert all(torch.equal(a, b * 0.25) for a, b in zip(gr, before))


@pytest.mark.parametrize("T,V,H", [(1, 5, 8), (700, 3, 264), (300, 5000, 8200), (257, 1, 4096)])
@pytest.mark.parametrize("fresh", [True, False])
def test_embedding_gradient(T, V, H, fresh):
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(T)
    ids = torch.randint(0, V, (T,), generator=g, device="cuda")
    gy = torch.randn(T, H, generator=g, device="cuda").bfloat16()
    mg = torch.randn(V, H, generator=g, device="cuda")
    want = (torch.zeros_like(mg) if fresh else mg).double().index_add(0, ids, gy.double())
    ops._ext.ext().embedding_grad(ids, gy, mg, fresh)
    assert (mg.double() - want).abs().max() <= 2.0 ** -23 * T * 8          # fp32 sums of at most T terms of size 4


@pytest.mark.parametrize("V", [8, 257, 2040, 32000, 50257])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_vocabulary_loss(V, dtype):
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(V)
    x = (3 * torch.randn(37, V, generator=g, device="cuda")).to(dtype)
    x[1, :V // 2] = -math.inf                                              # masked columns, whole packets of them first
    tgt = torch.randint(V // 2, V, (37,), generator=g, device="cuda")
    stats = ops.cross_entropy.ce_stats(x, tgt, 0)
    lse = stats[:, 0] + torch.log(stats[:, 1])
    want = torch.logsumexp(x.double(), -1)
    assert (lse.double() - want).abs().max() < 2e-5
    assert torch.equal(stats[:, 2], x.gather(1, tgt[:, None])[:, 0].float())
    gout = torch.rand(37, generator=g, device="cuda")
    got = ops.cross_entropy.ce_backward(x, tgt, lse, gout, 0, 0.0, V)
    ref = (torch.softmax(x.double(), -1) - torch.nn.functional.one_hot(tgt, V)) * gout[:, None].double()
    assert (got.double() - ref).abs().max() <= (2.0 ** -8 if dtype == torch.bfloat16 else 2e-5)


# NaN ends in the loss wherever it stands: alone in a packet, beside masked columns, behind them, in rows of one packet
@pytest.mark.parametrize("V", [8, 40, 2048, 4096, 5003])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_vocabulary_loss_of_nan(V, dtype):
    from neuronx_distributed_b200 import ops
    from neuronx_distributed_b200.parallel_layers.loss_functions import parallel_cross_entropy

    _groups()
    g = torch.Generator(device="cuda").manual_seed(V)
    x = torch.randn(7, V, generator=g, device="cuda").to(dtype)
    x[0, :8] = math.nan
    x[1, :8] = -math.inf
    x[1, 5] = math.nan
    x[2, :V // 2] = -math.inf
    x[2, V // 2] = math.nan
    x[3, V - 1] = math.nan
    x[4] = math.nan
    x[5, :V // 2] = -math.inf                               # masked, no NaN
    tgt = torch.full((7,), V - 2, device="cuda")
    stats = ops.cross_entropy.ce_stats(x, tgt, 0)
    want = [True] * 5 + [False] * 2
    assert stats[:, 1].isnan().tolist() == want
    loss = parallel_cross_entropy(x.unsqueeze(1), tgt.unsqueeze(1)).flatten()
    assert loss.isnan().tolist() == want
    ref = torch.nn.functional.cross_entropy(x[5:].double(), tgt[5:], reduction="none")
    assert (loss[5:].double() - ref).abs().max() < 2e-5


def test_vocabulary_loss_of_foreign_targets():
    """Targets that are no column of this shard, however far away, subtract nothing."""
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(6, 4096, generator=g, device="cuda")
    tgt = torch.tensor([-1, -100, 4096, 2 ** 32 + 3, -2 ** 63, 2 ** 63 - 1], device="cuda")
    stats = ops.cross_entropy.ce_stats(x, tgt, 0)
    assert not stats[:, 2].any()
    got = ops.cross_entropy.ce_backward(x, tgt, torch.logsumexp(x, -1), torch.ones(6, device="cuda"), 0, 0.0, 4096)
    assert (got.double() - torch.softmax(x.double(), -1)).abs().max() <= 2e-5


# chunks are 4096 elements; slices: fp32 arrays at `offset` elements, 16-bit ones at 2 or 4 more or fewer
@pytest.mark.parametrize("sizes", [[4095], [4096, 4097, 8192], [3] * 50 + [12289]])
@pytest.mark.parametrize("offset", [(0, 0), (0, 4), (4, 4), (4, 2), (1, 1)])
@pytest.mark.parametrize("gdtype,ldtype", [(torch.bfloat16, torch.bfloat16), (torch.float32, torch.bfloat16), (torch.float16, torch.float32),
                                           (torch.float32, None)])
def test_optimizer_slices(sizes, offset, gdtype, ldtype):
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(len(sizes))
    whole = []

    def arrays(dtype, at):
        whole.append([torch.rand(n + 16, generator=g, device="cuda").to(dtype) for n in sizes])
        return [t[at:at + n] for t, n in zip(whole[-1], sizes)]

    p, m, v = (arrays(torch.float32, offset[0]) for _ in range(3))
    gr = arrays(gdtype, offset[1])
    low = arrays(ldtype, offset[1]) if ldtype is not None else None
    outside = [[t.clone() for t in w] for w in whole]
    want = []
    scale, lr, b1, b2, eps, wd, step = 0.5, 1e-2, 0.9, 0.99, 1e-6, 0.1, 3
    for a, gg, c, d in zip(p, gr, m, v):
        a, c, d, gg = a.double(), c.double(), d.double(), gg.double() * scale
        c, d = b1 * c + (1 - b1) * gg, b2 * d + (1 - b2) * gg * gg
        want.append(((a - lr * math.sqrt(1 - b2 ** step) / (1 - b1 ** step) * c / (d.sqrt() + eps)) * (1 - lr * wd), c, d))
    ops.optim.fused_adamw_(p, gr, m, v, lr, b1, b2, eps, wd, step, torch.tensor(scale, device="cuda"), low)
    for i, w in enumerate(want):
        for a, b in zip((p[i], m[i], v[i]), w):             # a few fp32 roundings
            assert ((a.double() - b).abs() <= 2.0 ** -18 * (1 + b.abs())).all()
        assert low is None or torch.equal(low[i], p[i].to(ldtype))
    for w, o, at in zip(whole, outside, [offset[0]] * 3 + [offset[1]] * 2):
        for a, b, n in zip(w, o, sizes):
            assert torch.equal(a[:at], b[:at]) and torch.equal(a[at + n:], b[at + n:])


@pytest.mark.parametrize("n", [(1 << 20) - 1, 1 << 20, (1 << 20) + 13, 5 * 1000 * 1003])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("offset", [0, 1, 8])
def test_gradients_into_the_buffer(n, dtype, offset):
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(n)
    grad = torch.randn(n + offset, generator=g, device="cuda").to(dtype)[offset:]
    whole = torch.randn(n + 32, generator=g, device="cuda")
    buf, outside = whole[16:16 + n], whole.clone()
    want = buf + grad                                       # one fp32 sum per element
    ops.optim.grad_to_buffer_(buf, grad, True)
    assert torch.equal(buf, want)
    ops.optim.grad_to_buffer_(buf, grad, False)
    assert torch.equal(buf, grad.float())
    assert torch.equal(whole[:16], outside[:16]) and torch.equal(whole[16 + n:], outside[16 + n:])
    with pytest.raises(RuntimeError):
        ops.optim.grad_to_buffer_(buf, grad[:n - 1], False)
