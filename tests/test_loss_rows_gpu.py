"""Loss of rows that hold the whole vocabulary: edges of the packet groups, both block sizes, rows of another alignment, masked rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,V", [(3, 1), (5, 7), (700, 8), (400, 8192), (400, 8200), (300, 10001), (297, 16384), (2, 65536), (400, 65544)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_loss_of_whole_rows(rows, V, dtype):
    from neuronx_distributed_b200.ops import cross_entropy as ce

    g = torch.Generator(device="cuda").manual_seed(V)
    x = (3 * torch.randn(rows, V, generator=g, device="cuda")).to(dtype)
    t = torch.randint(0, V, (rows,), generator=g, device="cuda")
    x[0, : V // 2] = float("-inf")
    x[1, t[1]] = 30.0
    loss, lse = ce.ce_loss(x, t)
    want = torch.logsumexp(x.double(), -1)
    # terms: an argument of up to 60 rounded twice (2^-24 each), the exponential's 2^-22; sums of at most 300 terms per thread in fp32
    tol = 60 * 2.0 ** -23 + 2.0 ** -22 + 300 * 2.0 ** -24
    assert (lse.double() - want).abs().max() <= tol + 2.0 ** -23 * want.abs().max()
    picked = x.double().gather(1, t[:, None])[:, 0]
    finite = picked.isfinite()
    assert (loss.double() - (want - picked))[finite].abs().max() <= tol + 2.0 ** -22 * (want.abs() + picked.abs())[finite].max()
    assert (loss[~finite] == float("inf")).all()
    bad = x.clone()
    bad[-1, V - 1] = float("nan")
    bad[0] = float("-inf")
    loss, lse = ce.ce_loss(bad, t)
    assert lse[-1].isnan() and lse[0] == float("-inf") and loss[0].isnan()
    assert torch.equal(lse[1:-1], ce.ce_loss(x, t)[1][1:-1])
