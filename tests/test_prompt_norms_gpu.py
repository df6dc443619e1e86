"""Prompts of served models: residual sums inside the norms against the separate sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _served(hidden, heads, dtype, layers=2, batch=1, seq=32):
    import torch.distributed as dist

    from neuronx_distributed_b200.models.llama import LlamaConfig
    from neuronx_distributed_b200.models.llama_inference import LlamaForInference
    from neuronx_distributed_b200.parallel_layers import parallel_state as ps

    if not dist.is_initialized():
        dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1)
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(tensor_model_parallel_size=1)
    torch.manual_seed(0)
    cfg = LlamaConfig(vocab_size=64, hidden_size=hidden, intermediate_size=256, num_hidden_layers=layers, num_attention_heads=heads,
                      num_key_value_heads=1, max_position_embeddings=seq, dtype=dtype, device=torch.device("cuda"))
    m = LlamaForInference(cfg, batch_size=batch, max_seq_len=seq, on_device_sampling=False).eval()
    with torch.no_grad():
        for p in m.lm.parameters():
            if p.dim() == 2:
                p.copy_(torch.randn_like(p) * p.shape[1] ** -0.5)
    return m


def _prompt(model, ids):
    logits = model.context_encoding(ids, torch.full((ids.shape[0],), ids.shape[1] - 1, device="cuda"))
    n = ids.shape[1]
    return [logits] + [c[:, :n].clone() for c in [*model.kv.k, *model.kv.v]]


def _separate_sums(model, ids):
    """The same prompt with a hook on a norm: hooks see the module's own call, so the sums are made outside the norms."""
    handle = model._core.norm.register_forward_hook(lambda *a: None)
    try:
        return _prompt(model, ids)
    finally:
        handle.remove()


@pytest.mark.parametrize("H", [8, 1024, 2056, 4100, 8192, 8200, 16384, 20488])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_sum_and_norm_of_any_width(H, dtype):
    from neuronx_distributed_b200 import ops

    if H % (16 // dtype.itemsize):
        pytest.skip("the norm takes whole 16-byte packets")
    g = torch.Generator(device="cuda").manual_seed(H)
    x, r, w = (torch.randn(*s, generator=g, device="cuda").to(dtype) for s in ((5, H), (5, H), (H,)))
    with torch.no_grad():
        y, h = ops.norm.add_rms_norm(x, r, w, 1e-5)
        assert torch.equal(h, x + r) and torch.equal(y, ops.norm.rms_norm(x + r, w, 1e-5))


# widths whose norms do not fit the registers of a block: 1024 packets of 16 bytes
@pytest.mark.parametrize("hidden,heads,dtype", [(8320, 65, torch.bfloat16), (4224, 33, torch.float32)])
def test_prompt_of_wide_model(hidden, heads, dtype):
    m = _served(hidden, heads, dtype, layers=1)
    ids = torch.randint(0, 64, (1, 20), device="cuda")
    for a, b in zip(_prompt(m, ids), _separate_sums(m, ids)):
        assert torch.equal(a, b)


# up to eight rows the output projection adds the residual to its fp32 sum and rounds once, as token generation does
@pytest.mark.parametrize("batch,seq", [(1, 1), (2, 3), (1, 8), (4, 2), (1, 9), (2, 12)])
def test_short_prompts_round_once(batch, seq):
    m = _served(512, 4, torch.bfloat16, batch=batch)
    ids = torch.randint(0, 64, (batch, seq), device="cuda")
    for a, b in zip(_prompt(m, ids), _separate_sums(m, ids)):
        assert torch.equal(a, b)


def test_watched_norms_are_called():
    """A hook on all modules and a forward of one module's own see every norm of a prompt."""
    from neuronx_distributed_b200.modules.rms_norm import RMSNorm

    m = _served(256, 2, torch.bfloat16)
    ids = torch.randint(0, 64, (1, 16), device="cuda")
    seen = []
    for register in (torch.nn.modules.module.register_module_forward_hook, torch.nn.modules.module.register_module_forward_pre_hook):
        seen.clear()
        handle = register(lambda mod, *a: seen.append(mod) if isinstance(mod, RMSNorm) else None)
        try:
            _prompt(m, ids)
        finally:
            handle.remove()
        assert len(seen) == 2 * 2 + 1
    n = m._core.layers[1].input_layernorm
    seen.clear()
    n.forward = lambda x: (seen.append(n), type(n).forward(n, x))[1]
    _prompt(m, ids)
    assert len(seen) == 1


def test_attention_block_of_a_subclass():
    """A class with an attention block of its own gets the stream and gives it back with the block's output added."""
    m = _served(256, 2, torch.bfloat16)
    ids = torch.randint(0, 64, (1, 16), device="cuda")
    want, plain, calls = _prompt(m, ids), type(m), []

    def block(self, i, layer, x, positions, prefill, kv_len, tree=None):
        calls.append(i)
        return plain._attn_block(self, i, layer, x, positions, prefill, kv_len, tree)

    m.__class__ = type("Own", (plain,), {"_attn_block": block})
    for a, b in zip(_prompt(m, ids), want):
        assert torch.equal(a, b)
    assert calls == [0, 1]
