"""Normalised affinities are differentiated twice: the node around the kernels against the chain of plain operations, its two launches replaced by
plain code with the kernels' results."""
import types

import pytest
import torch

from dist_utils import run_distributed


def _kernels():
    def chain(aff, idx):
        a = aff * torch.zeros_like(aff).scatter_(1, idx, 1.0)
        return a / a.sum(-1, keepdim=True).clamp(min=1e-9)

    def moe_normalize(aff, idx):
        with torch.no_grad():
            return chain(aff, idx)

    def moe_normalize_grad(g, aff, idx):
        with torch.enable_grad():
            leaf = aff.detach().requires_grad_()
            return torch.autograd.grad(chain(leaf, idx), leaf, g.detach())[0]

    return types.SimpleNamespace(moe_normalize=moe_normalize, moe_normalize_grad=moe_normalize_grad)


def _penalty(module, path, x, logits, idx, strided):
    """The output, its first gradients, and the gradients of the squared norm of the first."""
    x, logits = x.clone().requires_grad_(), logits.clone().requires_grad_()
    aff = torch.softmax(logits, -1)
    if strided:
        aff = aff.t().contiguous().t()
    y = getattr(module, path)(x, aff, idx)
    first = torch.autograd.grad(y.square().sum(), (x, logits), create_graph=True)
    second = torch.autograd.grad(sum(g.square().sum() for g in first), (x, logits))
    return [y.detach(), *(g.detach() for g in first), *second]


def _cases(rank, world):
    from neuronx_distributed_b200 import ops
    from neuronx_distributed_b200.modules.moe import ExpertMLPsV2, RoutedExpertsMLPOpsConfig
    from neuronx_distributed_b200.ops import _ext
    from neuronx_distributed_b200.parallel_layers import parallel_state as ps

    ps.initialize_model_parallel(tensor_model_parallel_size=1)
    torch.manual_seed(0)
    T, E, k, H = 24, 6, 2, 16
    x, logits = torch.randn(T, H), torch.randn(T, E)
    idx = logits.topk(k, -1).indices
    plain, kernels = (ops.moe_blocks.normalize_ok, _ext.ext), _kernels()
    for act, glu in (("gelu", False), ("gelu", True), ("silu", True)):
        cfg = RoutedExpertsMLPOpsConfig(num_experts=E, top_k=k, hidden_size=H, intermediate_size=32, hidden_act=act, glu_mlp=glu,
                                        capacity_factor=2.0, normalize_top_k_affinities=True)
        m = ExpertMLPsV2(cfg).train()
        for path in ("forward_all_experts", "forward_capacity_factor"):
            for strided in (False, True):
                want = _penalty(m, path, x, logits, idx, strided)
                try:
                    ops.moe_blocks.normalize_ok, _ext.ext = (lambda aff, i: True), (lambda: kernels)
                    got = _penalty(m, path, x, logits, idx, strided)
                finally:
                    ops.moe_blocks.normalize_ok, _ext.ext = plain
                for a, b in zip(got, want):        # the same sums in 32 bits, in another order
                    assert (a - b).norm() <= 1e-5 * b.norm(), (act, glu, path, strided)


def test_second_derivatives_through_the_experts():
    run_distributed(_cases, 1)


@pytest.mark.parametrize("scale", [1.0, 1e-11])
def test_against_the_chain(monkeypatch, scale):
    """Rows in 64 bits, an expert chosen twice among them; below the least sum the quotient has one gradient less."""
    from neuronx_distributed_b200.ops import _ext, moe_blocks

    kernels = _kernels()
    monkeypatch.setattr(_ext, "ext", lambda: kernels)
    torch.manual_seed(1)
    aff = ((torch.rand(3, 5, dtype=torch.float64) + 0.5) * scale).requires_grad_()
    idx, go = torch.tensor([[0, 1], [4, 2], [3, 3]]), torch.randn(3, 5, dtype=torch.float64, requires_grad=True)
    mask = torch.zeros_like(aff).scatter_(1, idx, 1.0)
    results = []
    for w in (moe_blocks.normalize(aff, idx), aff * mask / (aff * mask).sum(-1, keepdim=True).clamp(min=1e-9)):
        (g,) = torch.autograd.grad(w.square().sum() + (w * go).sum(), aff, create_graph=True)
        results.append([w, g, *torch.autograd.grad(g.square().sum(), (aff, go))])
    for a, b in zip(*results):
        torch.testing.assert_close(a, b, rtol=1e-12, atol=1e-12 * float(b.abs().max()))
