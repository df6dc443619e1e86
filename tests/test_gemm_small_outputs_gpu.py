"""Products of fewer rows than the CTA pair's tile, on whichever kernel takes them: all three transposes, stored and accumulated, nothing
written behind the last row, the same bits from run to run."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(M, N, K, trans_a, trans_b, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randn((K, M) if trans_a else (M, K), generator=g, device="cuda").bfloat16()
    b = torch.randn((N, K) if trans_b else (K, N), generator=g, device="cuda").bfloat16()
    return a, b


@pytest.mark.parametrize("M", [8, 64, 120, 128, 136, 200, 248])
@pytest.mark.parametrize("N,K", [(264, 72), (1024, 2048), (520, 8192)])      # without and with the tail's split of K
@pytest.mark.parametrize("trans_a,trans_b", [(False, True), (False, False), (True, False)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_products_of_few_rows(M, N, K, trans_a, trans_b, dtype):
    from neuronx_distributed_b200 import ops

    a, b = _operands(M, N, K, trans_a, trans_b)
    x, y = (a.t() if trans_a else a).double(), (b.t() if trans_b else b).double()
    want, size = x @ y, x.abs() @ y.abs()
    for accumulate in (False, True):
        whole = torch.full((M + 1, N), 3.0, device="cuda", dtype=dtype)
        out = whole[:M]
        assert ops.gemm.matmul(a, b, trans_a, trans_b, out=out, accumulate=accumulate) is out
        assert (whole[M] == 3).all()
        ref = want + 3 * accumulate
        # K exact products and the old value summed in fp32 (each sum and each cut of the tensor cores at most 2^-23), then the type's rounding
        bound = (K + 1) * 2.0 ** -23 * (size + 3) + (2.0 ** -8 * ref.abs() if dtype == torch.bfloat16 else 0)
        assert ((out.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("M,N,K", [(128, 4096, 8192), (248, 512, 16384), (64, 1024, 4096), (8, 264, 8192)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_the_same_bits_every_time(M, N, K, accumulate):
    from neuronx_distributed_b200 import ops

    a, b = _operands(M, N, K, True, False, seed=1)
    first = None
    for _ in range(20):
        out = torch.full((M, N), 0.3, device="cuda")
        ops.gemm.matmul(a, b, True, False, out=out, accumulate=accumulate)
        first = out if first is None else first
        assert torch.equal(out, first)


def test_one_rule_in_both_languages():
    from neuronx_distributed_b200 import ops

    native = ops._ext._C.native
    for M in (1, 8, 127, 128, 129, 136, 255, 256, 5000):
        for N in (8, 16376, 16384, 16385, 16392, 128256):
            assert native.pairs(M, N) == ops.gemm._pairs(M, N)
