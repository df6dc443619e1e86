"""RMSNorm of few and of many rows (weights asked for early, or not), narrow, at the edge of the registers and beyond it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 64, 65])
@pytest.mark.parametrize("H", [8, 264, 8192, 8200, 12288])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_norm_rows(rows, H, dtype):
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(H)
    x = torch.randn(rows, H, generator=g, device="cuda").to(dtype)
    w = (1 + 0.1 * torch.randn(H, generator=g, device="cuda")).to(dtype)
    d = x.double()
    want = d * torch.rsqrt((d * d).mean(-1, keepdim=True) + 1e-5) * w.double()
    # fp32 sum of H squares per row and three roundings, then one to the type
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -19
    assert (ops.norm.rms_norm(x, w, 1e-5).double() - want).abs().max() <= tol * float(want.abs().max())
