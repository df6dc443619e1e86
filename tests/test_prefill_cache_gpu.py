"""Rotation of a prompt straight into the caches against the separate rotations and copies: the same bits, nothing written beyond the prompt."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("B,S,H,K,D", [(1, 1, 1, 1, 16), (1, 1000, 40, 40, 128), (2, 37, 8, 1, 128), (3, 64, 5, 5, 64)])
def test_rows_in_the_caches(B, S, H, K, D, dtype):
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(S)
    qkv = torch.randn(S, B, (H + 2 * K) * D, generator=g, device="cuda").to(dtype)
    q, k, v = (t.unflatten(-1, (-1, D)).transpose(0, 1) for t in qkv.split([H * D, K * D, K * D], -1))
    cos, sin = ops.rope.rope_tables(S + 5, D, device="cuda")
    kc, vc = (torch.full((B + 1, S + 3, K, D), 7.0, device="cuda", dtype=dtype) for _ in range(2))
    got = ops._ext.ext().prefill_rope_kv(q, k, v, cos, sin, kc, vc)
    assert torch.equal(got, ops.rope.apply_rotary(q, cos[:S], sin[:S]))
    assert torch.equal(kc[:B, :S], ops.rope.apply_rotary(k, cos[:S], sin[:S])) and torch.equal(vc[:B, :S], v)
    for c in (kc, vc):
        assert (c[B] == 7).all() and (c[:, S:] == 7).all()


@pytest.mark.parametrize("batch,seq", [(1, 9), (2, 37), (1, 128)])
def test_prompt_is_the_same(batch, seq, monkeypatch):
    import torch.distributed as dist

    from neuronx_distributed_b200.models.llama import LlamaConfig
    from neuronx_distributed_b200.models.llama_inference import LlamaForInference
    from neuronx_distributed_b200.parallel_layers import parallel_state as ps

    if not dist.is_initialized():
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1, device_id=torch.device("cuda", 0))
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(tensor_model_parallel_size=1)
    torch.manual_seed(0)
    cfg = LlamaConfig(vocab_size=512, hidden_size=512, intermediate_size=1024, num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=2,
                      max_position_embeddings=128, dtype=torch.bfloat16, device=torch.device("cuda", 0))
    model = LlamaForInference(cfg, batch_size=batch, max_seq_len=128, on_device_sampling=False).eval()
    ids = torch.randint(0, 512, (batch, seq), device="cuda")
    out = []
    for own in (True, False):
        model.kv.reset()
        taken = []
        if own:
            inner = LlamaForInference._prefill_in_cache
            monkeypatch.setattr(LlamaForInference, "_prefill_in_cache", lambda *a: taken.append(inner(*a)) or taken[-1])
        else:
            monkeypatch.setattr(LlamaForInference, "_prefill_in_cache", lambda *a: False)
        logits = model.context_encoding(ids)
        assert not own or taken == [True, True]
        out.append([logits.clone(), *(t.clone() for t in model.kv.k + model.kv.v)])
    for a, b in zip(*out):
        assert torch.equal(a, b)


@pytest.mark.parametrize("seq,longest", [(37, 128), (200, 256), (130, 130)])
def test_old_rows_of_the_caches_are_never_used(seq, longest):
    import torch.distributed as dist

    from neuronx_distributed_b200.models.llama import LlamaConfig
    from neuronx_distributed_b200.models.llama_inference import LlamaForInference
    from neuronx_distributed_b200.parallel_layers import parallel_state as ps

    if not dist.is_initialized():
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1, device_id=torch.device("cuda", 0))
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(tensor_model_parallel_size=1)
    torch.manual_seed(0)
    cfg = LlamaConfig(vocab_size=512, hidden_size=512, intermediate_size=1024, num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=2,
                      max_position_embeddings=longest, dtype=torch.bfloat16, device=torch.device("cuda", 0))
    model = LlamaForInference(cfg, batch_size=2, max_seq_len=longest, on_device_sampling=False).eval()
    ids = torch.randint(0, 512, (2, seq), device="cuda")
    out = []
    for left_there in (0.0, float("nan"), float("inf")):
        for t in model.kv.k + model.kv.v:
            t.fill_(left_there)
        logits = model.context_encoding(ids)
        out.append([logits.clone(), *(t[:, :seq].clone() for t in model.kv.k + model.kv.v)])
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert torch.equal(a, b)


@pytest.mark.parametrize("seq", [1, 37, 130, 200, 256])
@pytest.mark.parametrize("order", ["bshd", "sbhd", "bhsd", "cache"])
def test_a_sequence_does_not_see_its_neighbours(order, seq):
    """Rows behind a sequence's last belong to others: NaN there (keys, values, queries, gradients) stays there, forward and backward."""
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(seq)

    def make(heads):
        shape = {"bshd": (2, seq, heads, 128), "sbhd": (seq, 2, heads, 128), "bhsd": (2, heads, seq, 128), "cache": (2, seq + 20, heads, 128)}[order]
        t = torch.randn(shape, generator=g, device="cuda").bfloat16()
        return {"bshd": t, "sbhd": t.transpose(0, 1), "bhsd": t.transpose(1, 2), "cache": t[:, :seq]}[order], t

    (q, qm), (k, km), (v, vm), (go, gm) = make(4), make(2), make(2), make(4)
    f = ops._ext.ext()

    def both():
        o, lse = f.flash_attn_fwd(q, k, v, True, 128 ** -0.5, True)
        return [o, *f.flash_attn_bwd(go, q, k, v, o, lse, True, 128 ** -0.5, True, None, 1)]

    want = [t[0].clone() for t in both()]
    keep = [t[0].clone() for t in (q, k, v, go)]
    for t, m, x in zip((q, k, v, go), (qm, km, vm, gm), keep):
        m.fill_(float("nan"))
        t[0] = x
    for i, (a, b) in enumerate(zip(both(), want)):
        if i == 1:                                         # dQ: sums over K/V tiles arrive in any order: fp32, then one rounding to bf16
            assert (a[0].double() - b.double()).abs().max() <= 2.0 ** -7 * b.double().abs().max()
        else:
            assert torch.equal(a[0], b)


@pytest.mark.parametrize("seq", [1, 130])
@pytest.mark.parametrize("form", ["heads repeated", "sequences repeated", "one sequence of a batch", "one head of many", "slices of a projection", "every other row"])
def test_views_as_their_copies(form, seq):
    """Strides of 0, of dimensions of one and within a row: the maps give what a dense copy gives, forward and backward."""
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(seq)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()

    def make(h):
        if form == "heads repeated":
            return rnd(2, seq, 1, 128).expand(2, seq, h, 128)
        if form == "sequences repeated":
            return rnd(1, seq, h, 128).expand(2, seq, h, 128)
        if form == "one sequence of a batch":
            return rnd(3, seq + 5, h, 128)[1:2, 2:seq + 2]
        if form == "one head of many":
            return rnd(2, seq, 3 * h, 128)[:, :, 2:3]
        if form == "slices of a projection":
            return rnd(seq, 2, (h + 3) * 128)[..., 256:256 + h * 128].unflatten(-1, (h, 128)).transpose(0, 1)
        return rnd(2, 2 * seq, h, 128)[:, ::2]

    q, k, v, go = make(4), make(2), make(2), make(4)
    f = ops._ext.ext()
    res = []
    for dense in (False, True):
        a, b, c, d = (t.contiguous() if dense else t for t in (q, k, v, go))
        o, lse = f.flash_attn_fwd(a, b, c, True, 128 ** -0.5, True)
        res.append([o, lse, *f.flash_attn_bwd(d, a, b, c, o, lse, True, 128 ** -0.5, True, None, 1)])
    for i, (a, b) in enumerate(zip(*res)):
        if i == 2:                                         # dQ: sums over K/V tiles arrive in any order: fp32, then one rounding to bf16
            assert (a.double() - b.double()).abs().max() <= 2.0 ** -7 * b.double().abs().max()
        else:
            assert torch.equal(a, b)
