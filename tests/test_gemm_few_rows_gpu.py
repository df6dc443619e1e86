"""GEMM of few rows at the edges of its tiles, splits and rings."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 3, 8, 16, 17, 127, 128, 129, 256])
@pytest.mark.parametrize("N,K", [(8, 8), (128, 64), (136, 520), (1000, 4096), (4096, 200)])
@pytest.mark.parametrize("split", [0, 2, 8])
def test_rows(M, N, K, split):
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(M)
    x, w = (torch.randn(n, K, generator=g, device="cuda").bfloat16() for n in (M, N))
    got = ops._ext.ext().gemm_few_rows(x, w, split).double()
    want = x.double() @ w.double().t()
    # fp32 sums and one rounding to bfloat16
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -20 * K).all()


@pytest.mark.parametrize("M", [2, 3, 8])
def test_residual(M):
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(M)
    x, w, r = (torch.randn(*s, generator=g, device="cuda").bfloat16() for s in ((M, 5120), (6144, 5120), (M, 6144)))
    got = ops._ext.ext().gemv(x, w, r).double()
    want = x.double() @ w.double().t() + r.double()
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -20 * 5120).all()


# both sides of the rules that choose a kernel: rows, columns and length of the rows
@pytest.mark.parametrize("M", [2, 3, 4, 8, 64, 72, 128, 136, 176, 184])
@pytest.mark.parametrize("N,K", [(512, 512), (64, 4096), (264, 2048), (1032, 1016), (9480, 2048), (65544, 128)])
def test_rules(M, N, K):
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(M)
    x, w = (torch.randn(n, K, generator=g, device="cuda").bfloat16() for n in (M, N))
    got = ops.gemm.matmul(x, w, False, True)
    want = x.double() @ w.double().t()
    # fp32 sums over K terms, one rounding to bfloat16 (2^-9)
    assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -20 * K).all()
