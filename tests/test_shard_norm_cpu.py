"""What the squared norm of a sharded optimizer hands to its kernel: one list on one device and one tensor-parallel rank, else one of each kind."""
from types import SimpleNamespace

import pytest
import torch


@pytest.mark.parametrize("devices,lists", [(("cuda:0", "cuda:0"), [["sharded", "dup"]]), (("cuda:0", "cuda:1"), [["sharded"], ["dup"]])])
def test_lists_hold_tensors_of_one_device(monkeypatch, devices, lists):
    from neuronx_distributed_b200 import ops
    from neuronx_distributed_b200.optimizer.zero_redundancy_optimizer import Zero1Optimizer

    class Shard:                                           # a shard that says where it lies; no device is needed
        def __init__(self, name):
            self.name = name

        def __getitem__(self, _):
            return self

    def group(name, device):
        slot = SimpleNamespace(param=SimpleNamespace(shared=False, tensor_model_parallel=name == "sharded"))
        return SimpleNamespace(device=torch.device(device), grad_shard=Shard(name), shard_slices=lambda: [(slot, 0, 0, 4)])

    seen = []
    monkeypatch.setattr(ops.optim, "multi_tensor_sq_norm", lambda ts: seen.append([t.name for t in ts]) or SimpleNamespace(to=lambda dev: torch.ones(())))
    fake = SimpleNamespace(flat_groups=[group("sharded", devices[0]), group("dup", devices[1])])
    assert Zero1Optimizer._shard_sq_norm(fake) == len(lists) and seen == lists
