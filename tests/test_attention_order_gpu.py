"""Forward attention waits for its products in order: many work items per SM, where the softmax warps of a block drift apart."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(q, k, v):
    n, group = q.shape[1], q.shape[2] // k.shape[2]
    k, v = (t.float().repeat_interleave(group, 2).transpose(1, 2) for t in (k, v))
    s = q.float().transpose(1, 2) @ k.transpose(-1, -2) / math.sqrt(q.shape[-1])
    s = s.masked_fill(torch.ones(n, n, dtype=torch.bool, device=s.device).triu(1), -math.inf)
    return (torch.softmax(s, -1) @ v).transpose(1, 2)


# bf16 probabilities and outputs: 2^-9 relative each, averaged over the keys; an output row that misses one tile's product is off
# by its own size
@pytest.mark.parametrize("batch,seq,heads,kv_heads", [(2, 2048, 32, 32), (4, 1024, 32, 8), (8, 500, 32, 32), (8, 130, 64, 8)])
def test_same_rows_on_every_call(batch, seq, heads, kv_heads):
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v = (torch.randn(seq, batch, h, 128, generator=g, device="cuda").bfloat16().transpose(0, 1) for h in (heads, kv_heads, kv_heads))
    first = ops.attention.flash_attention(q, k, v, causal=True)
    for b in range(batch):
        want = _reference(q[b:b + 1], k[b:b + 1], v[b:b + 1])
        off = (first[b:b + 1].float() - want).norm(dim=-1) / want.norm(dim=-1)
        assert off.max() < 0.02
    for _ in range(20):
        assert torch.equal(ops.attention.flash_attention(q, k, v, causal=True), first)


# one query tile (blocks of 128 rows), tiles split between two streams (few tiles) and pairs of tiles with an odd one left
@pytest.mark.parametrize("batch,seq,heads,kv_heads", [(1, 1, 2, 1), (1, 127, 2, 2), (2, 129, 4, 2), (1, 640, 3, 3), (1, 1100, 16, 2), (3, 385, 40, 8),
                                                      (1, 700, 40, 40)])
def test_edges_of_tiles(batch, seq, heads, kv_heads):
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(seq)
    q, k, v = (torch.randn(seq, batch, h, 128, generator=g, device="cuda").bfloat16().transpose(0, 1) * s
               for h, s in ((heads, 4), (kv_heads, 1), (kv_heads, 1)))
    got, lse = ops._ext.ext().flash_attn_fwd(q, k, v, True, 128 ** -0.5, True)
    want = _reference(q, k, v)
    assert ((got.float() - want).norm(dim=-1) <= 0.02 * want.norm(dim=-1) + 1e-3).all()
    kf = k.float().repeat_interleave(heads // kv_heads, 2).transpose(1, 2)
    s = q.float().transpose(1, 2) @ kf.transpose(-1, -2) / math.sqrt(128)
    s = s.masked_fill(torch.ones(seq, seq, dtype=torch.bool, device=s.device).triu(1), -math.inf)
    assert (lse - torch.logsumexp(s, -1)).abs().max() < 1e-3


@pytest.mark.parametrize("sq,skv,heads", [(64, 1000, 4), (300, 65, 40), (257, 257, 100)])
def test_all_keys_visible(sq, skv, heads):
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(sq)
    q, k, v = (torch.randn(1, n, heads, 128, generator=g, device="cuda").bfloat16() for n in (sq, skv, skv))
    got = ops.attention.flash_attention(q, k, v, causal=False).float()
    p = torch.softmax(q.float().transpose(1, 2) @ k.float().transpose(1, 2).transpose(-1, -2) / math.sqrt(128), -1)
    want = (p @ v.float().transpose(1, 2)).transpose(1, 2)
    assert ((got - want).norm(dim=-1) <= 0.02 * want.norm(dim=-1) + 1e-3).all()


@pytest.mark.parametrize("batch", [1, 2])
def test_no_keys_is_an_error(batch):
    from neuronx_distributed_b200 import ops

    q, k = (torch.randn(batch, n, 8, 128, device="cuda").bfloat16() for n in (40, 0))
    with pytest.raises(RuntimeError):
        ops.attention.flash_attention(q, k, k, causal=False)
