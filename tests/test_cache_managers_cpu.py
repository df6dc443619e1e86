"""A served model works with a cache manager of another kind, through the manager's own calls alone."""
import torch

from dist_utils import run_distributed


class _Elsewhere:
    """Keeps its rows in one tensor a layer; no lists of key and value caches."""

    def __init__(self, layers, batch, longest, heads, dim):
        self.rows = [torch.zeros(2, batch, longest, heads, dim) for _ in range(layers)]
        self.kv_quant, self.seq_shards = None, 1

    def write_prefill(self, layer, k, v, seq_ids=None):
        self.rows[layer][:, :k.shape[0], :k.shape[1]] = torch.stack([k, v])

    def write_decode(self, layer, k, v, positions):
        self.rows[layer][:, torch.arange(k.shape[0]), positions] = torch.stack([k[:, 0], v[:, 0]])

    def get(self, layer, length=None):
        return self.rows[layer][0][:, :length], self.rows[layer][1][:, :length]

    def reset(self):
        for t in self.rows:
            t.zero_()


def _serve(rank, world):
    from neuronx_distributed_b200.models.llama import LlamaConfig
    from neuronx_distributed_b200.models.llama_inference import LlamaForInference
    from neuronx_distributed_b200.parallel_layers import parallel_state as ps

    ps.initialize_model_parallel(tensor_model_parallel_size=world)
    torch.manual_seed(0)
    cfg = LlamaConfig(vocab_size=64, hidden_size=32, intermediate_size=64, num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=2,
                      dtype=torch.float32, max_position_embeddings=32)
    m = LlamaForInference(cfg, batch_size=2, max_seq_len=32).eval()
    ids = torch.randint(0, 64, (2, 8))
    want = m.generate(ids, 4)
    m.kv = _Elsewhere(2, 2, 32, 2, 8)
    assert torch.equal(m.generate(ids, 4), want)


def test_manager_of_another_kind():
    run_distributed(_serve, 1, timeout=120)
