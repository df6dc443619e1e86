"""Backward of the norms at the edges of their blocks: one and two packets per thread, more and fewer rows than blocks."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,H", [(1, 8), (3, 264), (700, 1024), (150, 4096), (2500, 4104), (130, 8192), (600, 2048)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("residual", [False, True])
def test_norm_backward(rows, H, dtype, residual):
    from neuronx_distributed_b200 import ops

    if dtype == torch.float32 and H > 4096:
        pytest.skip("rows of more than 1024 packets are refused")
    g = torch.Generator(device="cuda").manual_seed(H)
    x, r, gy, gh = (torch.randn(rows, H, generator=g, device="cuda").to(dtype) for _ in range(4))
    w = (1 + 0.1 * torch.randn(H, generator=g, device="cuda")).to(dtype)
    ins = [t.clone().requires_grad_() for t in (x, r, w)]
    ref = [t.detach().double().requires_grad_() for t in (x, r, w)]
    if residual:
        got = torch.autograd.grad(ops.norm.add_rms_norm(*ins, 1e-5), ins, (gy, gh))
        h = ref[0] + ref[1]
        h = h + (h.detach().to(dtype).double() - h.detach())            # the stored sum
        want = torch.autograd.grad((h * torch.rsqrt((h * h).mean(-1, keepdim=True) + 1e-5) * ref[2], h), ref, (gy.double(), gh.double()))
    else:
        got = torch.autograd.grad(ops.norm.rms_norm(ins[0], ins[2], 1e-5), (ins[0], ins[2]), gy)
        h = ref[0]
        want = torch.autograd.grad(h * torch.rsqrt((h * h).mean(-1, keepdim=True) + 1e-5) * ref[2], (ref[0], ref[2]), gy.double())
    # fp32 sums over the row and over the rows, one rounding to the type
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -17
    for a, b in zip(got, want):
        assert a.dtype == dtype and (a.double() - b).abs().max() <= tol * max(1.0, float(b.abs().max()))
