"""Attention at the edges of its tiles, both directions, against 64-bit mathematics: one row, a tile less, exactly and one more than one of
queries (64 rows backward, 128 forward) and of keys (128), groups of heads with and without several blocks per KV head."""
import math

import pytest
import torch

from neuronx_distributed_b200 import ops

pytestmark = pytest.mark.gpu


def _reference(q, k, v, go, causal):
    q, k, v = (t.double().requires_grad_(True) for t in (q, k, v))
    group = q.shape[2] // k.shape[2]
    kk, vv = (t.repeat_interleave(group, 2) for t in (k, v))
    s = torch.einsum("bqhd,bkhd->bhqk", q, kk) / math.sqrt(128)
    if causal:
        s = s.masked_fill(torch.ones(s.shape[-2:], dtype=torch.bool, device=s.device).triu(1), -math.inf)
    o = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, -1), vv)
    return [o.detach(), *torch.autograd.grad(o, (q, k, v), go.double())]


def _check(B, S, Skv, H, K, causal, scale_q=1.0):
    g = torch.Generator(device="cuda").manual_seed(S * 131 + H)
    make = lambda s, h: torch.randn(s, B, h, 128, generator=g, device="cuda").bfloat16().transpose(0, 1)
    q, k, v, go = make(S, H) * scale_q, make(Skv, K), make(Skv, K), make(S, H)
    want = _reference(q, k, v, go, causal)
    q, k, v = (t.requires_grad_(True) for t in (q, k, v))
    o = ops.attention.flash_attention(q, k, v, causal=causal)
    got = [o, *torch.autograd.grad(o, (q, k, v), go)]
    for name, a, b in zip(("o", "dq", "dk", "dv"), got, want):
        # probabilities, their gradients, the output and the stored result are each rounded to bf16 once: four roundings of at most 2^-9; a
        # gradient that is zero in 64 bits (one key) is a difference of numbers of the size of go . v
        err = float((a.double() - b).norm() / b.norm().clamp(min=1e-2 * math.sqrt(b.numel())))
        assert err < 4 * 2 ** -9, (name, err)


@pytest.mark.parametrize("S", [1, 2, 63, 64, 65, 127, 128, 129, 191, 193, 256, 257, 385])
def test_causal_rows(S):
    _check(2, S, S, 4, 2, True)


@pytest.mark.parametrize("S,Skv", [(1, 300), (64, 129), (129, 64), (200, 127), (65, 1), (300, 128)])
def test_full_rows(S, Skv):
    _check(1, S, Skv, 3, 3, False)


@pytest.mark.parametrize("B,S,H,K", [(1, 200, 16, 1), (1, 513, 32, 8), (1, 130, 64, 8), (3, 129, 48, 8), (1, 1030, 8, 8), (4, 640, 40, 40)])
def test_heads(B, S, H, K):
    _check(B, S, S, H, K, True)


@pytest.mark.parametrize("scale", [0.01, 30.0])
def test_flat_and_steep_probabilities(scale):
    """Rows whose maximum hardly moves, and rows whose maximum jumps from tile to tile by more than the accumulator's spare range."""
    _check(1, 700, 700, 4, 4, True, scale)


def test_scores_that_are_no_numbers():
    """NaN and infinite keys or queries make NaN rows where they are seen, and only there."""
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = (torch.randn(1, 450, 2, 128, generator=g, device="cuda").bfloat16() for _ in range(3))
    want = ops.attention.flash_attention(q, k, v, causal=True)
    for value in (math.nan, math.inf):
        for row in (0, 130, 300, 449):
            k2, q2 = k.clone(), q.clone()
            k2[0, row, 1, 5] = value
            o = ops.attention.flash_attention(q, k2, v, causal=True)
            assert torch.equal(o[:, :, 0], want[:, :, 0]) and torch.equal(o[:, :row, 1], want[:, :row, 1])
            seen = q[0, row:, 1, 5] > 0 if value == math.inf else torch.ones(450 - row, dtype=torch.bool, device="cuda")
            assert o[0, row:, 1][seen].isnan().all()                   # q . k is NaN or +inf; where it is -inf the key has no weight
            q2[0, row, 1, 5] = math.nan
            o = ops.attention.flash_attention(q2, k, v, causal=True)
            rest = torch.arange(450, device="cuda") != row
            assert o[0, row, 1].isnan().all() and torch.equal(o[:, rest], want[:, rest])
