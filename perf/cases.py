"""Performance cases: the work that training and serving programs have this package do, through its public entry points.

Each case is a plain dict; ``prepare`` builds what a program holds before the call (weights, inputs, caches, graphs), ``run`` is one
pass, ``work`` counts the bytes and operations that the pass cannot do without, ``exact`` recomputes it in 64 bits with plain torch.
Sizes are those of the models in ``models/`` (Llama-2 7B / 13B / 70B, Mixtral, DBRX), of the smoke model, and of tensor-parallel
shards of them; weights and tokens are random.
"""
from __future__ import annotations

import math

import torch

DEVICE = "cuda"
BF16 = torch.bfloat16

# (hidden, intermediate) of dense feed-forward blocks: smoke model, 7B, 13B, one of eight tensor-parallel shards of 70B
MLP_SIZES = ((1024, 2816), (4096, 11008), (5120, 13824), (8192, 3584))
# (query heads, key/value heads): 7B, 13B, 70B, Mixtral, DBRX, one of four shards of 7B; head size 128 throughout
HEADS = ((32, 32), (40, 40), (64, 8), (32, 8), (48, 8), (8, 8))
# (experts, experts per token, hidden, intermediate): a quarter of Mixtral's and of DBRX's expert width (tensor-parallel shards)
MOE_SIZES = ((8, 2, 4096, 3584), (16, 4, 6144, 2688))
VOCABS = (32000, 32016, 100352)
HIDDEN = (1024, 2048, 4096, 5120, 6144, 8192)


def _model(hidden, intermediate, heads, kv_heads, vocab, layers):
    return {"hidden": hidden, "intermediate": intermediate, "heads": heads, "kv_heads": kv_heads, "vocab": vocab, "layers": layers}


SMALL = _model(1024, 2816, 8, 8, 4096, 2)            # the smoke model
LLAMA_7B = _model(4096, 11008, 32, 32, 32000, 2)     # two of its 32 layers
LLAMA_13B = _model(5120, 13824, 40, 40, 32016, 2)    # two of its 40 layers
LLAMA_70B_TP8 = _model(8192, 3584, 8, 1, 4000, 2)    # two layers of one of eight tensor-parallel shards


def listed():
    return [
        # one optimizer step of pre-training: forward, backward into fp32 gradients, clipping, AdamW on fp32 masters
        {"name": "train_step_7b", "kind": "train_step", "batch": 1, "seq": 2048, **LLAMA_7B},
        # the same program at the size of a unit test or a debugging run: launches and host time count
        {"name": "train_step_small", "kind": "train_step", "batch": 2, "seq": 512, **SMALL},
        # attention of the pre-training step: micro-batch of two sequences
        {"name": "attention_train", "kind": "attention", "batch": 1, "seq": 2048, "heads": 32, "kv_heads": 32, "backward": True},
        # attention of a prompt of no round length, grouped key/value heads
        {"name": "attention_prompt", "kind": "attention", "batch": 1, "seq": 1531, "heads": 64, "kv_heads": 8, "backward": False},
        # dense feed-forward block of the pre-training step
        {"name": "mlp_train", "kind": "mlp", "tokens": 4096, "hidden": 4096, "intermediate": 11008, "backward": True},
        # dense feed-forward block over a speculation window or a few short prompts
        {"name": "mlp_few_tokens", "kind": "mlp", "tokens": 48, "hidden": 4096, "intermediate": 11008, "backward": False},
        # residual sum and norm between the blocks, both directions
        {"name": "add_norm_train", "kind": "add_norm", "rows": 8192, "hidden": 4096},
        # vocabulary loss and the gradient of its logits
        {"name": "loss_train", "kind": "loss", "tokens": 4096, "vocab": 32000},
        # routed experts without dropped tokens, both directions
        {"name": "moe_train", "kind": "moe", "tokens": 4096, "experts": 8, "top_k": 2, "hidden": 4096, "intermediate": 3584},
        # a prompt of no round length through a served model: logits of its last token, key/value cache filled
        {"name": "prompt_13b", "kind": "prompt", "batch": 1, "seq": 1000, "cache": 2048, **LLAMA_13B},
        # one generated token of a served model, batch 1, as a captured program
        {"name": "token_13b", "kind": "token", "batch": 1, "cache": 2048, **LLAMA_13B},
        # attention of one generated token per sequence, a batch of long conversations
        {"name": "attention_token", "kind": "attention_token", "batch": 8, "heads": 32, "kv_heads": 8, "cache": 8192},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train_step", "attention", "attention", "mlp", "mlp", "add_norm", "loss", "moe", "prompt", "token",
                       "attention_token"])
    if kind == "train_step":
        batch = rng.choice([1, 2])
        return {"kind": kind, "batch": batch, "seq": 8 * _log_uniform(rng, 16, 250 // batch), **rng.choice([SMALL, SMALL, LLAMA_7B])}
    if kind == "attention":
        heads, kv_heads = rng.choice(HEADS)
        seq = _log_uniform(rng, 65, 65536 // heads)
        return {"kind": kind, "batch": rng.randint(1, max(1, min(4, 65536 // heads // seq))), "seq": seq, "heads": heads,
                "kv_heads": kv_heads, "backward": rng.random() < 0.5}
    if kind == "mlp":
        hidden, intermediate = rng.choice(MLP_SIZES)
        backward = rng.random() < 0.5
        tokens = 8 * _log_uniform(rng, 16, 512) if backward else _log_uniform(rng, 9, 2048)
        return {"kind": kind, "tokens": tokens, "hidden": hidden, "intermediate": intermediate, "backward": backward}
    if kind == "add_norm":
        return {"kind": kind, "rows": _log_uniform(rng, 64, 16384), "hidden": rng.choice(HIDDEN)}
    if kind == "loss":
        return {"kind": kind, "tokens": _log_uniform(rng, 128, 4096), "vocab": rng.choice(VOCABS)}
    if kind == "moe":
        experts, top_k, hidden, intermediate = rng.choice(MOE_SIZES)
        return {"kind": kind, "tokens": _log_uniform(rng, 512, 4096), "experts": experts, "top_k": top_k, "hidden": hidden,
                "intermediate": intermediate}
    if kind == "prompt":
        model = rng.choice([LLAMA_7B, LLAMA_13B, LLAMA_70B_TP8])
        batch = rng.choice([1, 2])
        return {"kind": kind, "batch": batch, "seq": _log_uniform(rng, 100, 1600 // batch), "cache": 2048, **model}
    if kind == "token":
        model = rng.choice([LLAMA_7B, LLAMA_13B, LLAMA_70B_TP8])
        return {"kind": kind, "batch": rng.randint(1, 8), "cache": 128 * _log_uniform(rng, 4, 32), **model}
    heads, kv_heads = rng.choice(HEADS)
    return {"kind": kind, "batch": rng.randint(1, 16), "heads": heads, "kv_heads": kv_heads, "cache": _log_uniform(rng, 256, 8192)}


# ---------------------------------------------------------------------------------------------------------------- inputs
def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    return g


def _normal(g, *shape, std=1.0, dtype=BF16):
    return (torch.randn(*shape, generator=g, device=DEVICE, dtype=torch.float32) * std).to(dtype)


def _draws(case, seed):
    """All random tensors of a case, from the seed alone; ``prepare`` hands them to the package, ``exact`` to plain torch."""
    g, kind, c = _generator(seed), case["kind"], case
    if kind == "attention":
        # v is a slice of the fused projection's output, q and k come from the rotation: [S, B, heads, 128] in memory, used as [B, S, ...]
        S, B, H, K = c["seq"], c["batch"], c["heads"], c["kv_heads"]
        q = _normal(g, S, B, H, 128).transpose(0, 1)
        k = _normal(g, S, B, K, 128).transpose(0, 1)
        v = _normal(g, S, B, (H + 2 * K) * 128)[..., (H + K) * 128:].unflatten(-1, (K, 128)).transpose(0, 1)
        return {"q": q, "k": k, "v": v, "go": _normal(g, S, B, H, 128).transpose(0, 1)}
    if kind == "mlp":
        T, H, I = c["tokens"], c["hidden"], c["intermediate"]
        return {"x": _normal(g, T, 1, H), "gate_up_proj": _normal(g, 2 * I, H, std=0.02), "down_proj": _normal(g, H, I, std=0.02),
                "go": _normal(g, T, 1, H, std=0.1)}
    if kind == "add_norm":
        R, H = c["rows"], c["hidden"]
        return {"x": _normal(g, R, 1, H), "r": _normal(g, R, 1, H, std=2.0), "w": 1 + _normal(g, H, std=0.1),
                "gy": _normal(g, R, 1, H), "gh": _normal(g, R, 1, H)}
    if kind == "loss":
        T, V = c["tokens"], c["vocab"]
        return {"logits": _normal(g, T, 1, V, std=2.0), "target": torch.randint(0, V, (T, 1), generator=g, device=DEVICE),
                "go": torch.full((T, 1), 1.0 / T, device=DEVICE)}
    if kind == "moe":
        T, E, k, H, I = c["tokens"], c["experts"], c["top_k"], c["hidden"], c["intermediate"]
        aff = torch.softmax(torch.randn(T, E, generator=g, device=DEVICE), -1)
        return {"x": _normal(g, T, H), "aff": aff, "index": aff.topk(k, -1).indices, "go": _normal(g, T, H, std=0.1),
                "gate_up_proj": _normal(g, E, H, 2 * I, std=0.02), "down_proj": _normal(g, E, I, H, std=0.02)}
    if kind == "attention_token":
        B, H, K, L = c["batch"], c["heads"], c["kv_heads"], c["cache"]
        return {"q": _normal(g, B, 1, H, 128), "k": _normal(g, B, L, K, 128), "v": _normal(g, B, L, K, 128),
                "positions": torch.randint(L // 2, L, (B,), generator=g, device=DEVICE)}
    # whole models
    H, I, V, nq, nkv = c["hidden"], c["intermediate"], c["vocab"], c["heads"] * 128, c["kv_heads"] * 128
    w = {"model.embed_tokens.weight": _normal(g, V, H), "model.norm.weight": 1 + _normal(g, H, std=0.1),
         "lm_head.weight": _normal(g, V, H, std=H ** -0.5)}
    for i in range(c["layers"]):
        p = f"model.layers.{i}."
        w[p + "input_layernorm.weight"] = 1 + _normal(g, H, std=0.1)
        w[p + "post_attention_layernorm.weight"] = 1 + _normal(g, H, std=0.1)
        w[p + "self_attn.qkv_proj.weight_qkv"] = _normal(g, nq + 2 * nkv, H, std=H ** -0.5)
        w[p + "self_attn.o_proj.weight"] = _normal(g, H, nq, std=nq ** -0.5)
        w[p + "mlp.gate_up_proj.weight"] = _normal(g, 2 * I, H, std=H ** -0.5)
        w[p + "mlp.down_proj.weight"] = _normal(g, H, I, std=I ** -0.5)
    out = {"weights": w}
    if kind == "token":
        B, L = c["batch"], c["cache"]
        out["ids"] = torch.randint(0, V, (B, 1), generator=g, device=DEVICE)
        out["positions"] = torch.randint(L // 2, L, (B,), generator=g, device=DEVICE)
        out["kv"] = [(_normal(g, B, L, c["kv_heads"], 128), _normal(g, B, L, c["kv_heads"], 128)) for _ in range(c["layers"])]
    else:
        out["ids"] = torch.randint(0, V, (c["batch"], c["seq"]), generator=g, device=DEVICE)
    return out


# ------------------------------------------------------------------------------------------------------- the package's state
TRAINING = {"optimizer_config": {"zero_one_enabled": True, "grad_clipping": True, "max_grad_norm": 1.0},
            "mixed_precision_config": {"use_master_weights": True, "use_fp32_grad_acc": True, "use_master_weights_in_ckpt": False}}
ADAM = {"lr": 1e-4, "betas": (0.9, 0.95), "eps": 1e-6, "weight_decay": 0.1}


def _package():
    """The package with its parallel groups up: one process, as in a program on one GPU."""
    import torch.distributed as dist

    import neuronx_distributed_b200 as nxd
    from neuronx_distributed_b200.parallel_layers import parallel_state as ps

    if not dist.is_initialized():
        torch.cuda.set_device(0)
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1, device_id=torch.device("cuda", 0))
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(tensor_model_parallel_size=1)
    return nxd


def _load(module, weights):
    own = module.state_dict()
    with torch.no_grad():
        for name, w in weights.items():
            own[name].copy_(w)


def _llama_config(case, seq):
    from neuronx_distributed_b200.models.llama import LlamaConfig

    return LlamaConfig(vocab_size=case["vocab"], hidden_size=case["hidden"], intermediate_size=case["intermediate"],
                       num_hidden_layers=case["layers"], num_attention_heads=case["hidden"] // 128,
                       num_key_value_heads=case["kv_heads"], max_position_embeddings=seq, dtype=BF16, device=torch.device("cuda", 0))


def _full_size(case):
    """Heads as the model's configuration wants them: a shard's case names fewer than hidden / 128."""
    return case["heads"] * 128 == case["hidden"]


def prepare(case, seed):
    nxd = _package()
    kind, d = case["kind"], _draws(case, seed)
    state = {"case": case, **d}
    if kind == "attention":
        if case["backward"]:
            for n in "qkv":
                state[n].requires_grad_(True)
    elif kind == "mlp":
        from neuronx_distributed_b200.models.llama import LlamaConfig, LlamaMLP
        from neuronx_distributed_b200.utils.adamw_fp32_optim_params import AdamW_FP32OptimParams

        cfg = LlamaConfig(hidden_size=case["hidden"], intermediate_size=case["intermediate"], dtype=BF16, device=torch.device("cuda", 0))
        mlp = LlamaMLP(cfg)
        _load(mlp, {"gate_up_proj.weight": state.pop("gate_up_proj"), "down_proj.weight": state.pop("down_proj")})
        state["mlp"] = mlp
        if case["backward"]:
            # the optimizer gives every weight its fp32 gradient buffer, which the backward pass writes
            config = nxd.neuronx_distributed_config(tensor_parallel_size=1, **TRAINING)
            state["optimizer"] = nxd.initialize_parallel_optimizer(config, AdamW_FP32OptimParams, mlp.parameters(), **ADAM)
            state["x"].requires_grad_(True)
    elif kind == "add_norm":
        for n in ("x", "r", "w"):
            state[n].requires_grad_(True)
    elif kind == "loss":
        state["logits"].requires_grad_(True)
    elif kind == "moe":
        from neuronx_distributed_b200.modules.moe import ExpertMLPsV2, RoutedExpertsMLPOpsConfig

        cfg = RoutedExpertsMLPOpsConfig(num_experts=case["experts"], top_k=case["top_k"], hidden_size=case["hidden"],
                                        intermediate_size=case["intermediate"], hidden_act="silu", glu_mlp=True, capacity_factor=None,
                                        normalize_top_k_affinities=True)
        experts = ExpertMLPsV2(cfg, dtype=BF16, device=torch.device("cuda", 0))
        _load(experts, {"mlp_op.gate_up_proj.weight": state.pop("gate_up_proj"), "mlp_op.down_proj.weight": state.pop("down_proj")})
        state["experts"] = experts.train()
        state["x"].requires_grad_(True)
        state["aff"].requires_grad_(True)
    elif kind == "train_step":
        from neuronx_distributed_b200.models.llama import LlamaForCausalLM
        from neuronx_distributed_b200.utils.adamw_fp32_optim_params import AdamW_FP32OptimParams

        config = nxd.neuronx_distributed_config(tensor_parallel_size=1, **TRAINING)
        model = nxd.initialize_parallel_model(config, lambda: LlamaForCausalLM(_llama_config(case, case["seq"])))
        _load(model.module, state.pop("weights"))
        state["model"] = model
        state["optimizer"] = nxd.initialize_parallel_optimizer(config, AdamW_FP32OptimParams, model.parameters(), **ADAM)
    elif kind in ("prompt", "token"):
        from neuronx_distributed_b200.models.llama_inference import LlamaForInference
        from neuronx_distributed_b200.trace.model_builder import ModelBuilder

        cfg = _llama_config(case, case["cache"])
        if not _full_size(case):
            cfg = _shard_config(cfg, case)
        model = LlamaForInference(cfg, batch_size=case["batch"], max_seq_len=case["cache"], on_device_sampling=False).eval()
        _load(model.lm, state.pop("weights"))
        state["model"] = model
        if kind == "prompt":
            state["last"] = torch.full((case["batch"],), case["seq"] - 1, dtype=torch.long, device=DEVICE)
        else:
            builder = ModelBuilder(tp_degree=1, use_cuda_graphs=True)
            builder.add("token_generation_model", model, [(state["ids"], state["positions"])],
                        step_fn=lambda m, ids, positions: m.token_generation(ids, positions))
            state["program"] = builder.trace()
            for (k, v), kc, vc in zip(state.pop("kv"), model.kv.k, model.kv.v):
                kc.copy_(k)
                vc.copy_(v)
    return state


def _shard_config(cfg, case):
    """One tensor-parallel rank's layer sizes in a model of its own: fewer heads than hidden / 128."""
    from dataclasses import dataclass

    from neuronx_distributed_b200.models.llama import LlamaConfig

    @dataclass
    class ShardConfig(LlamaConfig):
        @property
        def head_dim(self):
            return 128

    values = {f: getattr(cfg, f) for f in cfg.__dataclass_fields__}
    values["num_attention_heads"] = case["heads"]
    return ShardConfig(**values)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "attention":
        from neuronx_distributed_b200 import ops

        if not case["backward"]:
            with torch.no_grad():
                return ops.attention.flash_attention(state["q"], state["k"], state["v"], causal=True)
        o = ops.attention.flash_attention(state["q"], state["k"], state["v"], causal=True)
        return [o, *torch.autograd.grad(o, (state["q"], state["k"], state["v"]), state["go"])]
    if kind == "mlp":
        if not case["backward"]:
            with torch.no_grad():
                return state["mlp"](state["x"])
        state["optimizer"].zero_grad()
        state["x"].grad = None
        y = state["mlp"](state["x"])
        y.backward(state["go"])
        return [y, state["x"].grad, state["mlp"].gate_up_proj.weight.main_grad, state["mlp"].down_proj.weight.main_grad]
    if kind == "add_norm":
        from neuronx_distributed_b200 import ops

        y, h = ops.norm.add_rms_norm(state["x"], state["r"], state["w"], 1e-5)
        return [y, h, *torch.autograd.grad((y, h), (state["x"], state["r"], state["w"]), (state["gy"], state["gh"]))]
    if kind == "loss":
        from neuronx_distributed_b200.parallel_layers.loss_functions import parallel_cross_entropy

        loss = parallel_cross_entropy(state["logits"], state["target"])
        return [loss, *torch.autograd.grad(loss, (state["logits"],), state["go"])]
    if kind == "moe":
        e = state["experts"]
        y = e(state["x"], state["aff"], state["index"])
        return [y, *torch.autograd.grad(y, (state["x"], state["aff"], e.mlp_op.gate_up_proj.weight, e.mlp_op.down_proj.weight),
                                        state["go"])]
    if kind == "attention_token":
        from neuronx_distributed_b200 import ops

        with torch.no_grad():
            return ops.attention.decode_attention(state["q"], state["k"], state["v"], state["positions"])
    if kind == "train_step":
        state["optimizer"].zero_grad()
        loss = state["model"].run_train(input_ids=state["ids"], labels=state["ids"])
        state["optimizer"].step()
        params = dict(state["model"].module.named_parameters())
        return {"loss": loss, "grads": {n: p.main_grad for n, p in params.items()}, "weights": {n: p.data for n, p in params.items()}}
    if kind == "prompt":
        logits = state["model"].context_encoding(state["ids"], state["last"])
        S = case["seq"]
        return [logits, [k[:, :S] for k in state["model"].kv.k], [v[:, :S] for v in state["model"].kv.v]]
    return state["program"](state["ids"], state["positions"])


# ------------------------------------------------------------------------------------------------------------------- work
def _causal_pairs(seq):
    return seq * (seq + 1) // 2


def _model_params(c):
    nq, nkv = c["heads"] * 128, c["kv_heads"] * 128
    return c["layers"] * (c["hidden"] * (2 * nq + 2 * nkv) + 3 * c["hidden"] * c["intermediate"])


def work(case):
    c, kind = case, case["kind"]
    if kind == "attention":
        q, kv = c["batch"] * c["seq"] * c["heads"] * 128, c["batch"] * c["seq"] * c["kv_heads"] * 128
        products = 4.0 * c["batch"] * c["heads"] * _causal_pairs(c["seq"]) * 128
        if not c["backward"]:
            return {"bytes": 2 * (2 * q + 2 * kv), "flops": products}
        return {"bytes": 2 * (4 * q + 4 * kv), "flops": 3.5 * products}
    if kind == "mlp":
        n, x = 3 * c["hidden"] * c["intermediate"], c["tokens"] * c["hidden"]
        if not c["backward"]:
            return {"bytes": 2 * n + 4 * x, "flops": 2.0 * n * c["tokens"]}
        return {"bytes": 2 * n + 4 * n + 8 * x, "flops": 6.0 * n * c["tokens"]}
    if kind == "add_norm":
        return {"bytes": 2 * 7 * c["rows"] * c["hidden"], "flops": 0}
    if kind == "loss":
        return {"bytes": 2 * 2 * c["tokens"] * c["vocab"], "flops": 0}
    if kind == "moe":
        n, x = 3 * c["hidden"] * c["intermediate"], c["tokens"] * c["hidden"]
        return {"bytes": 2 * 2 * c["experts"] * n + 2 * 4 * x, "flops": 6.0 * n * c["tokens"] * c["top_k"]}
    if kind == "attention_token":
        # sequences stand at three quarters of the cache on average
        return {"bytes": 2 * 2 * c["batch"] * c["kv_heads"] * 128 * 0.75 * c["cache"], "flops": 0}
    body, head = _model_params(c), c["vocab"] * c["hidden"]
    if kind == "token":
        kv = 2 * 2 * c["layers"] * c["batch"] * c["kv_heads"] * 128 * 0.75 * c["cache"]
        return {"bytes": 2 * (body + head) + kv, "flops": 2.0 * c["batch"] * (body + head)}
    tokens = c["batch"] * c["seq"]
    products = 4.0 * c["layers"] * c["batch"] * c["heads"] * _causal_pairs(c["seq"]) * 128
    if kind == "prompt":
        return {"bytes": 2 * (body + head) + 2 * 2 * c["layers"] * tokens * c["kv_heads"] * 128,
                "flops": 2.0 * tokens * body + 2.0 * c["batch"] * head + products}
    # read and written once: bf16 weights, fp32 masters and two moments; fp32 gradients written once and read once
    n = body + 2 * head
    return {"bytes": n * (2 + 2 + 3 * 8 + 8), "flops": 6.0 * tokens * (body + head) + 3.5 * products}


# relative error (2-norm) that another correct implementation in bf16 would show: about four times the distance of each path from
# its 64-bit value (attention 0.0025, feed-forward 0.0035, norm and loss 0.0025, experts 0.005), less for whole models, where a
# rounding travels through every layer that follows (0.007 to 0.01 for logits and gradients)
TOLERANCE = {"attention": 0.01, "attention_token": 0.01, "mlp": 0.014, "add_norm": 0.01, "loss": 0.01, "moe": 0.02, "token": 0.025,
             "prompt": 0.03, "train_step": 0.03}


def tolerance(case):
    return {"rel": TOLERANCE[case["kind"]]}


# ------------------------------------------------------------------------------------------------------------ in 64 bits
def _silu(x):
    return x / (1 + torch.exp(-x))


def _rms(x, w, eps=1e-5):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _rotate(x, positions):
    """x [B, S, heads, 128], positions [B, S] or [S]: the two halves of a head are the real and imaginary parts."""
    # the angles are products of fp32 values in the package's tables; the frequencies are their fp32 values here too
    inv = 1.0 / (10000.0 ** (torch.arange(0, 128, 2, dtype=torch.float32, device=x.device) / 128))
    angle = positions.to(torch.float32).unsqueeze(-1) * inv
    c, s = torch.cos(angle.double()).unsqueeze(-2), torch.sin(angle.double()).unsqueeze(-2)
    a, b = x[..., :64], x[..., 64:]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


class _Causal(torch.autograd.Function):
    """Causal softmax attention in 64 bits, one head at a time in both directions."""

    @staticmethod
    def _head(q, k):
        s = (q @ k.transpose(-1, -2)) / math.sqrt(128)
        n = s.shape[-1]
        return torch.softmax(s.masked_fill_(torch.ones(n, n, dtype=torch.bool, device=s.device).triu_(1), -math.inf), -1)

    @staticmethod
    def forward(ctx, q, k, v):
        ctx.save_for_backward(q, k, v)
        group = q.shape[2] // k.shape[2]
        o = torch.empty_like(q)
        for h in range(q.shape[2]):
            o[:, :, h] = _Causal._head(q[:, :, h], k[:, :, h // group]) @ v[:, :, h // group]
        return o

    @staticmethod
    def backward(ctx, go):
        q, k, v = ctx.saved_tensors
        group = q.shape[2] // k.shape[2]
        gq, gk, gv = torch.empty_like(q), torch.zeros_like(k), torch.zeros_like(v)
        for h in range(q.shape[2]):
            j = h // group
            p, g = _Causal._head(q[:, :, h], k[:, :, j]), go[:, :, h]
            gp = g @ v[:, :, j].transpose(-1, -2)
            gs = p * (gp - (gp * p).sum(-1, keepdim=True)) / math.sqrt(128)
            gv[:, :, j] += p.transpose(-1, -2) @ g
            gq[:, :, h] = gs @ k[:, :, j]
            gk[:, :, j] += gs.transpose(-1, -2) @ q[:, :, h]
        return gq, gk, gv


def _mlp(x, gate_up, down):
    gate, up = (x @ gate_up.t()).chunk(2, -1)
    return (_silu(gate) * up) @ down.t()


def _token_attention(q, k, v, positions):
    B, L, K = k.shape[:3]
    G = q.shape[2] // K
    s = torch.einsum("bkgd,blkd->bkgl", q[:, 0].unflatten(1, (K, G)), k) / math.sqrt(128)
    hidden = torch.arange(L, device=k.device)[None, :] > positions[:, None]
    p = torch.softmax(s.masked_fill(hidden[:, None, None, :], -math.inf), -1)
    return torch.einsum("bkgl,blkd->bkgd", p, v).flatten(1, 2).unsqueeze(1)


def _layers(case, w, x, positions, attend):
    """Decoder layers and the last norm over x [B, S, hidden]; ``attend(layer, q, k, v)`` gets rotated q and k."""
    nq, nkv = case["heads"] * 128, case["kv_heads"] * 128
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        qkv = _rms(x, w[p + "input_layernorm.weight"]) @ w[p + "self_attn.qkv_proj.weight_qkv"].t()
        q, k, v = (t.unflatten(-1, (-1, 128)) for t in qkv.split([nq, nkv, nkv], -1))
        o = attend(i, _rotate(q, positions), _rotate(k, positions), v)
        x = x + o.flatten(-2) @ w[p + "self_attn.o_proj.weight"].t()
        x = x + _mlp(_rms(x, w[p + "post_attention_layernorm.weight"]), w[p + "mlp.gate_up_proj.weight"], w[p + "mlp.down_proj.weight"])
    return _rms(x, w["model.norm.weight"])


def exact(case, seed):
    kind, d = case["kind"], _draws(case, seed)
    f = {n: t.double() for n, t in d.items() if isinstance(t, torch.Tensor) and t.is_floating_point()}
    if kind == "attention":
        for t in f.values():
            t.requires_grad_(True)
        o = _Causal.apply(f["q"], f["k"], f["v"])
        if not case["backward"]:
            return o.detach()
        return [o.detach(), *torch.autograd.grad(o, (f["q"], f["k"], f["v"]), f["go"])]
    if kind == "mlp":
        if not case["backward"]:
            return _mlp(f["x"], f["gate_up_proj"], f["down_proj"])
        inputs = [f[n].requires_grad_(True) for n in ("x", "gate_up_proj", "down_proj")]
        y = _mlp(*inputs)
        return [y.detach(), *torch.autograd.grad(y, inputs, f["go"])]
    if kind == "add_norm":
        inputs = [f[n].requires_grad_(True) for n in ("x", "r", "w")]
        h = inputs[0] + inputs[1]
        y = _rms(h, inputs[2])
        return [y.detach(), h.detach(), *torch.autograd.grad((y, h), inputs, (f["gy"], f["gh"]))]
    if kind == "loss":
        logits = f["logits"].requires_grad_(True)
        loss = torch.logsumexp(logits, -1) - logits.gather(-1, d["target"].unsqueeze(-1)).squeeze(-1)
        return [loss.detach(), *torch.autograd.grad(loss, (logits,), f["go"])]
    if kind == "moe":
        inputs = [f[n].requires_grad_(True) for n in ("x", "aff", "gate_up_proj", "down_proj")]
        x, aff, w1, w2 = inputs
        chosen = torch.zeros_like(aff).scatter(1, d["index"], 1.0)
        a = aff * chosen
        a = a / a.sum(-1, keepdim=True)
        y = torch.zeros_like(x)
        for e in range(case["experts"]):
            rows = chosen[:, e].nonzero().squeeze(1)
            y = y.index_add(0, rows, _mlp(x[rows], w1[e].t(), w2[e].t()) * a[rows, e].unsqueeze(-1))
        return [y.detach(), *torch.autograd.grad(y, inputs, f["go"])]
    if kind == "attention_token":
        return _token_attention(f["q"], f["k"], f["v"], d["positions"])
    w = {n: t.double() for n, t in d["weights"].items()}
    if kind == "token":
        caches = [(k.double(), v.double()) for k, v in d["kv"]]
        rows = torch.arange(case["batch"], device=DEVICE)

        def attend(i, q, k, v):
            kc, vc = caches[i]
            kc[rows, d["positions"]], vc[rows, d["positions"]] = k[:, 0], v[:, 0]
            return _token_attention(q, kc, vc, d["positions"])

        h = _layers(case, w, w["model.embed_tokens.weight"][d["ids"]], d["positions"].unsqueeze(1), attend)
        return h[:, 0] @ w["lm_head.weight"].t()
    positions = torch.arange(case["seq"], device=DEVICE)
    if kind == "prompt":
        ks, vs = [], []

        def attend(i, q, k, v):
            ks.append(k)
            vs.append(v)
            return _Causal.apply(q, k, v)

        h = _layers(case, w, w["model.embed_tokens.weight"][d["ids"]], positions, attend)
        return [h[:, -1] @ w["lm_head.weight"].t(), ks, vs]
    for t in w.values():
        t.requires_grad_(True)
    h = _layers(case, w, w["model.embed_tokens.weight"][d["ids"]], positions, lambda i, q, k, v: _Causal.apply(q, k, v))
    logits = (h[:, :-1] @ w["lm_head.weight"].t()).flatten(0, 1)
    target = d["ids"][:, 1:].flatten()
    loss = (torch.logsumexp(logits, -1) - logits.gather(-1, target.unsqueeze(-1)).squeeze(-1)).mean()
    grads = dict(zip(w, torch.autograd.grad(loss, list(w.values()))))
    norm = torch.sqrt(sum((g * g).sum() for g in grads.values()))
    clip = min(1.0, 1.0 / (float(norm) + 1e-6))
    (b1, b2), lr = ADAM["betas"], ADAM["lr"]
    weights = {}
    for n, t in w.items():
        g = grads[n] * clip
        step = lr * math.sqrt(1 - b2) / (1 - b1)
        weights[n] = (t.detach() - step * (1 - b1) * g / (torch.sqrt((1 - b2) * g * g) + ADAM["eps"])) * (1 - lr * ADAM["weight_decay"])
    return {"loss": loss.detach(), "grads": grads, "weights": weights}
