"""Gradient of the token table of a model whose optimizer keeps fp32 gradient buffers: what autograd's own lookup gives."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _table(V, H, main_grad=True):
    import torch.distributed as dist

    from neuronx_distributed_b200.parallel_layers import parallel_state as ps
    from neuronx_distributed_b200.parallel_layers.layers import ParallelEmbedding

    if not dist.is_initialized():
        dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1)
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(tensor_model_parallel_size=1)
    torch.manual_seed(0)
    emb = ParallelEmbedding(V, H, device=torch.device("cuda"), dtype=torch.bfloat16)
    signals = []
    if main_grad:                                           # what the sharded optimizer does with a parameter
        w = emb.weight
        w.main_grad, w.main_grad_fresh = torch.full((V, H), 7.0, device="cuda"), True
        w._nxd_grad_ready = lambda p: signals.append(p.main_grad.clone())

        def accumulate(p):
            if p.main_grad_fresh:
                p.main_grad.copy_(p.grad)
            else:
                p.main_grad.add_(p.grad)
            p.main_grad_fresh, p.grad = False, None
            p._nxd_grad_ready(p)

        w.register_post_accumulate_grad_hook(accumulate)
    return emb, signals


def _sums(ids, gy, V):
    return torch.zeros(V, gy.shape[-1], device="cuda", dtype=torch.double).index_add(0, ids.flatten(), gy.flatten(0, -2).double())


def _close(got, want, terms):
    # fp32 sums of `terms` values of size 4, one rounding to bfloat16
    assert (got.double() - want).abs().max() <= 2.0 ** -8 * want.abs().max() + 2.0 ** -21 * terms


def test_one_signal_for_two_lookups():
    """A table used twice in a step is final when both uses are in: a bucket that is sent on the first signal would lose the second."""
    emb, signals = _table(50, 64)
    a, b = torch.randint(0, 50, (2, 9), device="cuda"), torch.randint(0, 50, (30,), device="cuda")
    ga, gb = torch.randn(2, 9, 64, device="cuda").bfloat16(), torch.randn(30, 64, device="cuda").bfloat16()
    torch.autograd.backward((emb(a), emb(b)), (ga, gb))
    assert len(signals) == 1
    _close(signals[0], _sums(a, ga, 50) + _sums(b, gb, 50), 48)


def test_hooks_and_direct_gradients():
    emb, signals = _table(40, 64)
    ids, gy = torch.randint(0, 40, (33,), device="cuda"), torch.randn(33, 64, device="cuda").bfloat16()
    mask = (torch.arange(40, device="cuda") % 2).unsqueeze(1)
    handle = emb.weight.register_hook(lambda g: g * mask)   # train some rows only
    emb(ids).backward(gy)
    want = _sums(ids, gy, 40)
    _close(signals[0], want * mask, 33)
    handle.remove()
    got, = torch.autograd.grad(emb(ids), emb.weight, gy)
    _close(got, want, 33)
    assert len(signals) == 1 and got.dtype == torch.bfloat16
    y = emb(ids)
    with torch.no_grad():
        emb.weight.mul_(0.5)                                # the table's values take no part in its gradient
    y.backward(gy)
    _close(signals[1], want * (1 + mask), 66)
    # twice differentiable, as the lookup is
    x = torch.randn(33, 64, device="cuda").bfloat16().requires_grad_()
    g, = torch.autograd.grad(emb(ids), emb.weight, x, create_graph=True)
    gg, = torch.autograd.grad(g.float().square().sum(), x)
    want = (2 * _sums(ids, x.detach(), 40))[ids]
    assert (gg.double() - want).norm() <= 2.0 ** -6 * want.norm()
    emb.collect_output = False                              # then a function transform goes through
    out = torch.vmap(lambda i: emb(i))(ids.view(3, 11))
    assert torch.equal(out, emb(ids).view(3, 11, 64))


# ids of one stretch of 64 tokens, of several, and of one more or fewer; on a vocabulary shard the tokens of other ranks all look up row 0
@pytest.mark.parametrize("T,V,H,repeat", [(64, 9, 8, 1.0), (65, 9, 2056, 1.0), (129, 2, 264, 0.5), (640, 3, 64, 0.0), (1025, 70, 128, 0.0),
                                          (4096, 500, 1024, 7 / 8), (4099, 500, 1032, 1.0), (32768, 100, 256, 7 / 8)])
def test_repeated_tokens(T, V, H, repeat):
    emb, _ = _table(V, H)
    g = torch.Generator(device="cuda").manual_seed(T)
    ids = torch.randint(0, V, (T,), generator=g, device="cuda")
    ids[torch.rand(T, generator=g, device="cuda") < repeat] = 1
    gy = torch.randn(T, H, generator=g, device="cuda").bfloat16()
    got, = torch.autograd.grad(emb(ids), emb.weight, gy)
    want = _sums(ids, gy, V)
    # fp32 sums of at most T values of size 4 (in stretches: their error grows with the square root), one rounding to bfloat16
    assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -23 * 8 * T).all()
    again, = torch.autograd.grad(emb(ids), emb.weight, gy)
    assert torch.equal(got, again)


def test_tokens_outside_the_table_add_nothing():
    from neuronx_distributed_b200 import ops

    ids = torch.tensor([-1] * 70 + [3] * 3 + [5, 2 ** 40, 6] + [2] * 70, device="cuda")
    gy = torch.randn(len(ids), 64, device="cuda").bfloat16()
    out = torch.ones(6, 64, device="cuda")
    ops._ext.ext().embedding_grad(ids, gy, out, False)
    ok = (ids >= 0) & (ids < 6)
    _close(out, 1 + _sums(ids[ok], gy[ok], 6), 70)


@pytest.mark.parametrize("shape", [(1,), (3, 257), (2, 4, 33)])
def test_lookups_with_and_without_python_in_their_node(shape):
    from neuronx_distributed_b200 import ops
    from neuronx_distributed_b200.parallel_layers.layers import _TableLookup

    g = torch.Generator(device="cuda").manual_seed(len(shape))
    w = torch.randn(500, 72, generator=g, device="cuda").bfloat16().requires_grad_()
    ids = torch.randint(0, 500, shape, generator=g, device="cuda")
    go = torch.randn(*shape, 72, generator=g, device="cuda").bfloat16()
    out = []
    for lookup in (_TableLookup.apply, ops._ext.ext().native.table_lookup):
        y = lookup(ids, w)
        out.append((y, *torch.autograd.grad(y, w, go.transpose(0, -1).contiguous().transpose(0, -1))))
    assert all(torch.equal(a, b) for a, b in zip(*out)) and torch.equal(out[0][0], w[ids])


def test_its_gradient_is_differentiated_again():
    """The gradient of the table is linear in the upstream one: with create_graph it keeps its graph, in both nodes."""
    from neuronx_distributed_b200 import ops
    from neuronx_distributed_b200.parallel_layers.layers import _TableLookup

    g = torch.Generator(device="cuda").manual_seed(9)
    w = torch.randn(40, 64, generator=g, device="cuda").bfloat16().requires_grad_()
    ids = torch.randint(0, 40, (3, 50), generator=g, device="cuda")
    go = torch.randn(3, 50, 64, generator=g, device="cuda").bfloat16().requires_grad_()
    second = []
    for lookup in (_TableLookup.apply, ops._ext.ext().native.table_lookup, lambda i, t: torch.nn.functional.embedding(i, t)):
        (gw,) = torch.autograd.grad(lookup(ids, w), w, go, create_graph=True)
        second.append(torch.autograd.grad(gw.float().square().sum(), go)[0])
    assert torch.equal(second[0], second[2]) and torch.equal(second[1], second[2]) and second[2].any()
