"""Single-token attention over a cache, at the edges of its tiles (16 rows a warp, 64 a block) and stretches."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(q, k, v, positions):
    out = torch.zeros(q.shape, device=q.device)
    group = q.shape[2] // k.shape[2]
    for b, p in enumerate(positions.tolist()):
        n = max(0, min(p + 1, k.shape[1]))
        if n == 0:
            continue
        kb, vb = (t[b, :n].float().repeat_interleave(group, 1) for t in (k, v))
        s = torch.einsum("hd,lhd->hl", q[b, 0].float(), kb) / math.sqrt(128)
        out[b, 0] = torch.einsum("hl,lhd->hd", torch.softmax(s, -1), vb)
    return out


@pytest.mark.parametrize("group", [1, 2, 4, 8])
@pytest.mark.parametrize("rows,positions", [(1, [0, 0]), (17, [15, 16]), (130, [63, 64]), (700, [-1, 699]), (2500, [2499, 40]),
                                            (64, [62, 5000])])
def test_edges(group, rows, positions):
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(rows + group)
    kv = torch.randn(2, rows, 2, 2 * 128, generator=g, device="cuda").bfloat16()      # k and v interleaved: strided views
    k, v = kv[..., :128], kv[..., 128:]
    q = torch.randn(2, 1, 2 * group, 128, generator=g, device="cuda").bfloat16() * 3
    pos = torch.tensor(positions, device="cuda")
    want = _reference(q, k, v, pos)
    for b, p in enumerate(positions):
        if 0 <= p + 1 < rows:
            kv[b, p + 1:] = math.nan                                               # rows behind the position are never used
    got = ops.attention.decode_attention(q, k, v, pos).float()
    # one rounding to bfloat16 (2^-9 of the value) over fp32 sums
    assert (got - want).abs().max() <= 2.0 ** -8 * want.abs().max()
    assert torch.isfinite(got).all()


def test_partial_results_merge_to_the_whole():
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = (torch.randn(2, n, h, 128, generator=g, device="cuda").bfloat16() for n, h in ((1, 8), (600, 2), (600, 2)))
    pos = torch.tensor([599, 250], device="cuda")
    whole = ops.attention.decode_attention(q, k, v, pos).float()[:, 0]
    parts = [ops._ext.ext().decode_attention_partial(q, k[:, a:a + 300], v[:, a:a + 300], pos - a, 128 ** -0.5) for a in (0, 300)]
    m = torch.maximum(parts[0][1][..., 0], parts[1][1][..., 0])
    num = sum(o * torch.exp(ml[..., 0] - m)[..., None] for o, ml in parts)
    den = sum(ml[..., 1] * torch.exp(ml[..., 0] - m) for _, ml in parts)
    assert (num / den[..., None] - whole).abs().max() <= 2.0 ** -8 * whole.abs().max()


@pytest.mark.parametrize("batch,kv_heads,group,rows", [(1, 1, 4, 4096), (1, 1, 8, 4097), (1, 1, 1, 8193), (1, 1, 2, 20000), (1, 40, 1, 2048), (4, 8, 4, 7000),
                                                      (16, 8, 8, 4096), (3, 37, 2, 511)])
def test_numbers_of_stretches(batch, kv_heads, group, rows):
    """Merges of 2 to 64 stretches (16 of them at once), launches of more and of fewer than three blocks per SM."""
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(rows)
    k, v = (torch.randn(batch, rows, kv_heads, 128, generator=g, device="cuda").bfloat16() for _ in range(2))
    q = torch.randn(batch, 1, kv_heads * group, 128, generator=g, device="cuda").bfloat16() * 2
    pos = torch.randint(rows // 2, rows, (batch,), generator=g, device="cuda")
    want = _reference(q, k, v, pos)
    got = ops.attention.decode_attention(q, k, v, pos).float()
    assert (got - want).abs().max() <= 2.0 ** -8 * want.abs().max()


@pytest.mark.parametrize("group", [3, 5, 6, 7])
@pytest.mark.parametrize("rows,positions", [(1, [0, 0]), (130, [63, 64]), (700, [300, 699]), (2500, [2499, 40])])
def test_groups_of_other_sizes(group, rows, positions):
    from neuronx_distributed_b200 import ops

    assert ops.attention.decode_group_ok(*(torch.empty(2, 1, n, 128, dtype=torch.bfloat16, device="cuda") for n in (2 * group, 2, 2)))
    test_edges(group, rows, positions)


def test_rows_that_are_no_packets_go_the_general_way():
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(7)
    k, v = (torch.randn(2, 200, 2, 132, generator=g, device="cuda").bfloat16()[..., 1:129] for _ in range(2))
    q = torch.randn(2, 1, 12, 128, generator=g, device="cuda").bfloat16()
    pos = torch.tensor([199, 60], device="cuda")
    want = _reference(q, k, v, pos)
    got = ops.attention.decode_attention(q, k, v, pos).float()
    assert not ops.attention.decode_group_ok(q, k, v) and (got - want).abs().max() <= 2.0 ** -7 * want.abs().max()      # general way: bf16 probabilities too


@pytest.mark.parametrize("group", [1, 2, 4, 8])
def test_such_rows_of_every_group(group):
    from neuronx_distributed_b200 import ops
    from neuronx_distributed_b200.models import llama_inference
    from neuronx_distributed_b200.modules.attention.flash_decode import _local_partial

    g = torch.Generator(device="cuda").manual_seed(group)
    q = torch.randn(2, 1, 2 * group, 128, generator=g, device="cuda").bfloat16()
    pos = torch.tensor([89, 60], device="cuda")
    rows = torch.randn(2, 2, 90, 2, 136, generator=g, device="cuda").bfloat16()
    for k, v in (rows[..., 4:132].unbind(), (rows[0, ..., :128], rows[1, ..., 1:129])):
        assert not ops.attention.decode_group_ok(q, k, v)
        want = _reference(q, k, v, pos)
        o, _, l = _local_partial(q, k, v, pos, 128 ** -0.5)
        for got in (ops.attention.decode_attention(q, k, v, pos), llama_inference._decode_attention(q, k, v, pos), (o / l[..., None]).unsqueeze(1)):
            assert (got.float() - want).abs().max() <= 2.0 ** -7 * want.abs().max()


@pytest.mark.parametrize("group", [3, 5, 6, 7])
def test_parts_of_groups_of_other_sizes(group):
    """A shard of a cache, as distributed decoding calls it: un-normalised output, row maximum and row sum."""
    from neuronx_distributed_b200 import ops
    from neuronx_distributed_b200.modules.attention.flash_decode import _local_partial

    g = torch.Generator(device="cuda").manual_seed(group)
    k, v = (torch.randn(2, 300, 2, 128, generator=g, device="cuda").bfloat16() for _ in range(2))
    q = torch.randn(2, 1, 2 * group, 128, generator=g, device="cuda").bfloat16()
    pos = torch.tensor([400, 70], device="cuda")
    before = ops._ext.launches()
    o, m, l = _local_partial(q, k, v, pos, 128 ** -0.5)
    assert ops._ext.launches() - before == 2
    want = _reference(q, k, v, pos)[:, 0]
    assert (o / l[..., None] - want).abs().max() <= 2.0 ** -8 * want.abs().max()
    s = torch.einsum("bhd,blhd->bhl", q[:, 0].float(), k.float().repeat_interleave(group, 2)) * 128 ** -0.5
    s[1, :, 71:] = -math.inf
    torch.testing.assert_close(m, s.amax(-1), rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("batch,kv_heads,group,rows", [(16, 8, 1, 2000), (16, 8, 2, 2000), (16, 8, 3, 1999), (16, 8, 5, 2001), (16, 8, 6, 2000), (16, 8, 7, 1900),
                                                      (8, 32, 1, 4096), (8, 32, 1, 8192)])
def test_launches_of_more_than_three_blocks_per_sm(batch, kv_heads, group, rows):
    """Two stages a warp: sequences of no row, of one, of a tile more or less, of every row, and of lengths in between."""
    from neuronx_distributed_b200 import ops

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert batch * kv_heads * min((6 * sms + batch * kv_heads - 1) // (batch * kv_heads), (rows + 255) // 256) > 3 * sms
    g = torch.Generator(device="cuda").manual_seed(rows + group)
    k, v = (torch.randn(batch, rows, kv_heads, 128, generator=g, device="cuda").bfloat16() for _ in range(2))
    q = torch.randn(batch, 1, kv_heads * group, 128, generator=g, device="cuda").bfloat16() * 2
    pos = torch.randint(0, rows, (batch,), generator=g, device="cuda")
    pos[:7] = torch.tensor([-1, 0, 63, 64, rows - 1, rows + 5, rows // 2])
    want = _reference(q, k, v, pos)
    for b, p in enumerate(pos.tolist()):
        k[b, p + 1:], v[b, p + 1:] = math.nan, math.nan                            # rows behind the position are never used
    got = ops.attention.decode_attention(q, k, v, pos).float()
    for b in range(batch):                                                         # one rounding to bfloat16 over fp32 sums
        assert (got[b] - want[b]).abs().max() <= 2.0 ** -8 * want[b].abs().max()
    o, ml = ops._ext.ext().decode_attention_partial(q, k, v, pos, 128 ** -0.5)
    o = torch.where(ml[..., 1:] > 0, o / ml[..., 1:], 0)
    assert (o - want[:, 0]).abs().max() <= 2.0 ** -8 * want.abs().max()
