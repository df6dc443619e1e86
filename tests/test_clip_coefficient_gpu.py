"""Norm and clipping coefficient in one launch: the bits of the operations that they stand for."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sq", [0.0, 1e-40, 1e-12, 0.3, 1.0, 1.000001, 2.0, 3e7, 3e38, float("inf"), float("nan")])
@pytest.mark.parametrize("max_norm", [1.0, 0.3, 1, 1e30])
def test_norm_and_coefficient(sq, max_norm):
    from neuronx_distributed_b200 import ops

    t = torch.tensor(sq, device="cuda")
    before = ops._ext.launches()
    norm, coeff = ops.optim.clip_coefficient(t, max_norm)
    assert ops._ext.launches() - before == 1 and norm.shape == coeff.shape == ()
    want = t.sqrt()
    torch.testing.assert_close(norm, want, rtol=0, atol=0, equal_nan=True)
    torch.testing.assert_close(coeff, torch.clamp(max_norm / (want + 1e-6), max=1.0), rtol=0, atol=0, equal_nan=True)
    host = ops.optim.clip_coefficient(t.cpu(), max_norm)               # CPU: the operations
    torch.testing.assert_close(coeff.cpu(), host[1], rtol=2 ** -22, atol=0, equal_nan=True)
