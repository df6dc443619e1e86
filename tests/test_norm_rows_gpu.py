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


@pytest.mark.parametrize("rows_per_sm", [0, 7, 8])        # one row; the last count with a packet a thread; the first with two
@pytest.mark.parametrize("dtype,H", [(torch.bfloat16, 4096), (torch.bfloat16, 4104), (torch.bfloat16, 6144), (torch.bfloat16, 6152),
                                     (torch.float32, 2052), (torch.float32, 3072)])
def test_norm_backward_rows(rows_per_sm, dtype, H):
    from neuronx_distributed_b200 import ops

    rows = max(1, rows_per_sm * torch.cuda.get_device_properties(0).multi_processor_count)
    g = torch.Generator(device="cuda").manual_seed(H)
    x, r, gy, gh = (torch.randn(rows, H, generator=g, device="cuda").to(dtype) for _ in range(4))
    w = (1 + 0.1 * torch.randn(H, generator=g, device="cuda")).to(dtype)
    x, r, w = (t.requires_grad_() for t in (x, r, w))
    y, h = ops.norm.add_rms_norm(x, r, w, 1e-5)
    dx, dr, dw = torch.autograd.grad((y, h), (x, r, w), (gy, gh))
    hd, wd = h.detach().double(), w.detach().double()      # the stored sum is what the norm sees
    rstd = torch.rsqrt((hd * hd).mean(-1, keepdim=True) + 1e-5)
    n, gw = hd * rstd, gy.double() * wd
    want = gh.double() + rstd * (gw - n * (gw * n).mean(-1, keepdim=True))
    want_w = (gy.double() * n).sum(0)
    # fp32 sums of H terms per row and of all rows per column in parts, then one rounding to the type
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -18
    assert torch.equal(dx, dr) and (dx.double() - want).abs().max() <= tol * want.abs().max()
    assert (dw.double() - want_w).abs().max() <= tol * want_w.abs().max()
    z = ops.norm.rms_norm(h.detach().requires_grad_(), w, 1e-5)
    dz = torch.autograd.grad(z, w, gy)[0]
    assert (dz.double() - want_w).abs().max() <= tol * want_w.abs().max()
