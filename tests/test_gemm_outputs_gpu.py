"""fp32 GEMM outputs at the edges of their tiles: stored, accumulated, and split over the tokens."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,M,N,accumulate", [(64, 256, 8, False), (136, 264, 40, True), (1000, 520, 264, False), (4096, 512, 1032, True),
                                                   (4096, 4096, 4096, False)])
def test_weight_gradients_in_fp32(tokens, M, N, accumulate):
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(tokens)
    dy, x = (torch.randn(tokens, n, generator=g, device="cuda").bfloat16() for n in (M, N))
    out = torch.randn(M + 1, N, generator=g, device="cuda")
    guard, want = out[M].clone(), dy.double().t() @ x.double() + (out[:M].double() if accumulate else 0)
    ops.gemm.matmul(dy, x, True, False, out=out[:M], accumulate=accumulate)
    # exact products, fp32 sums over `tokens` terms
    assert (out[:M].double() - want).abs().max() <= 2.0 ** -22 * tokens * dy.float().abs().max() * x.float().abs().max()
    assert torch.equal(out[M], guard)


@pytest.mark.parametrize("M,N,counts", [(64, 128, [1, 0, 3]), (320, 192, [2, 2, 0, 0]), (256, 64, [0, 5])])
@pytest.mark.parametrize("dtype,accumulate", [(torch.bfloat16, False), (torch.float32, False), (torch.float32, True)])
def test_grouped_weight_gradients(M, N, counts, dtype, accumulate):
    from neuronx_distributed_b200 import ops

    g, block = torch.Generator(device="cuda").manual_seed(M), 128
    seg = torch.cumsum(torch.tensor([0] + counts), 0).int()
    rows = int(seg[-1]) * block + 256
    x, dy = (torch.randn(rows, n, generator=g, device="cuda").bfloat16() for n in (M, N))
    out = torch.randn(len(counts), M, N, generator=g, device="cuda").to(dtype)
    want = out.double() if accumulate else torch.zeros(out.shape, device="cuda", dtype=torch.double)
    for e in range(len(counts)):
        a, b = int(seg[e]) * block, int(seg[e + 1]) * block
        want[e] += x[a:b].double().t() @ dy[a:b].double()
    ops._ext.ext().grouped_wgrad(x, dy, out, seg.cuda(), block, accumulate)
    # fp32 sums as above; one rounding to bfloat16 (2^-9) of the result
    assert (out.double() - want).abs().max() <= (2.0 ** -8 if dtype is torch.bfloat16 else 2.0 ** -16) * max(1.0, want.abs().max())


# a last round of few tiles is split along K and summed by a second kernel: ragged rows, columns and k-blocks, both output types; behind
# full rounds of 74 tiles (80 and 160 tiles) and alone; `tail`: the output types for which the plan splits it
@pytest.mark.parametrize("M,N,K,tail", [(1000, 5112, 2504, "bf16 fp32"), (1000, 5112, 4104, "bf16 fp32"), (2040, 5112, 4104, "bf16 fp32"),
                                        (264, 2056, 4096, "bf16"), (520, 1032, 2504, "bf16"), (256, 1024, 1024, ""), (1000, 5120, 1032, ""), (300, 264, 640, ""),
                                        (5000, 4104, 520, "")])
@pytest.mark.parametrize("dtype,accumulate", [(torch.bfloat16, False), (torch.bfloat16, True), (torch.float32, False), (torch.float32, True)])
@pytest.mark.parametrize("trans", [(False, True), (False, False), (True, False)])
def test_split_tail(M, N, K, tail, dtype, accumulate, trans):
    from neuronx_distributed_b200 import ops

    if trans[0] and M % 8:
        M += 8 - M % 8
    assert (ops._ext.ext().gemm_2cta_workspace(M, N, K, dtype is torch.float32, accumulate) > 0) == (("fp32" if dtype is torch.float32 else "bf16") in tail)
    g = torch.Generator(device="cuda").manual_seed(K)
    a = torch.randn(*((K, M) if trans[0] else (M, K)), generator=g, device="cuda").bfloat16()
    b = torch.randn(*((N, K) if trans[1] else (K, N)), generator=g, device="cuda").bfloat16()
    out = torch.randn(M + 1, N, generator=g, device="cuda").to(dtype)
    guard = out[M].clone()
    want = (a.double().t() if trans[0] else a.double()) @ (b.double().t() if trans[1] else b.double())
    if accumulate:
        want = want + out[:M].double()
    ops._ext.ext().gemm_bf16_2cta(a, b, out[:M], trans[0], trans[1], accumulate)
    # fp32 sums over K terms; one rounding to bfloat16
    assert (out[:M].double() - want).abs().max() <= (2.0 ** -8 if dtype is torch.bfloat16 else 0) * want.abs().max() + 2.0 ** -20 * K
    assert torch.equal(out[M], guard)


# the kernel that sums a split tail writes whole groups of 8 columns: products of other widths are not split
@pytest.mark.parametrize("N", [4, 5116])
@pytest.mark.parametrize("accumulate", [False, True])
def test_no_tail_for_other_widths(N, accumulate):
    from neuronx_distributed_b200 import ops

    e, M, K = ops._ext.ext(), 1000, 2504
    assert e.gemm_2cta_workspace(M, 5112, K, True, accumulate) > 0 and e.gemm_2cta_workspace(M, N, K, True, accumulate) == 0
    g = torch.Generator(device="cuda").manual_seed(N)
    a, b = (torch.randn(n, K, generator=g, device="cuda").bfloat16() for n in (M, N))
    out = torch.randn(M + 1, N, generator=g, device="cuda")
    guard, want = out[M].clone(), a.double() @ b.double().t() + (out[:M].double() if accumulate else 0)
    e.gemm_bf16_2cta(a, b, out[:M], False, True, accumulate)
    assert (out[:M].double() - want).abs().max() <= 2.0 ** -20 * K      # fp32 sums over K terms
    assert torch.equal(out[M], guard)


def test_output_views_of_any_alignment():
    """TMA wants 16-byte aligned outputs; views that are not get their result by way of a buffer, added to them in fp32."""
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(5)
    for dtype in (torch.float32, torch.bfloat16):
        for N in (16, 264):
            a, b = (torch.randn(n, 72, generator=g, device="cuda").bfloat16() for n in (320, N))
            flat = torch.zeros(320 * N + 2, device="cuda", dtype=dtype)
            for accumulate in (False, True):
                out = flat[1:-1].view(320, N)
                assert ops.gemm.matmul(a, b, trans_b=True, out=out, accumulate=accumulate) is out
            want = 2 * (a.double() @ b.double().t())
            # fp32 sums over 72 terms; stored and added to, each with one rounding to bfloat16 (2^-9)
            assert (out.double() - want).abs().max() <= (2.0 ** -8 if dtype is torch.bfloat16 else 2.0 ** -18) * want.abs().max()
            assert flat[0] == 0 and flat[-1] == 0


# more parts than pairs of SMs: the tail (48 tiles in 3 parts each) itself takes several rounds
@pytest.mark.parametrize("M,N,K", [(704, 4096, 11008), (700, 4088, 11016)])
@pytest.mark.parametrize("trans", [(False, True), (False, False)])
def test_tail_of_many_parts(M, N, K, trans):
    from neuronx_distributed_b200 import ops

    e = ops._ext.ext()
    assert e.gemm_2cta_workspace(M, N, K, False, False) > 0
    g = torch.Generator(device="cuda").manual_seed(N)
    a = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    b = torch.randn(*((N, K) if trans[1] else (K, N)), generator=g, device="cuda").bfloat16()
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    e.gemm_bf16_2cta(a, b, out, trans[0], trans[1], False)
    want = a.double() @ (b.double().t() if trans[1] else b.double())
    assert (out.double() - want).abs().max() <= 2.0 ** -8 * want.abs().max() + 2.0 ** -20 * K       # fp32 sums over K terms, one rounding
    again = torch.empty_like(out)
    e.gemm_bf16_2cta(a, b, again, trans[0], trans[1], False)
    assert torch.equal(out, again)


def test_parts_of_a_tail_are_bounded():
    """The fp32 workspace of a product is at most three parts of 256 KB for each pair of SMs, however long K is; one beyond that is shared out
    otherwise and is right."""
    import random

    from neuronx_distributed_b200 import ops

    e, rng = ops._ext.ext(), random.Random(3)
    bound = 3 * (torch.cuda.get_device_properties(0).multi_processor_count // 2) * 256 * 256 * 4
    sizes = [(1000, 4096, 128256), (2048, 4096, 22016), (3584, 1024, 28672), (3000, 4096, 32000)]
    sizes += [(8 * rng.randint(16, 1024), 128 * rng.randint(1, 256), 64 * rng.randint(4, 4096)) for _ in range(2000)]
    taken = [e.gemm_2cta_workspace(*size, f32, add) for size in sizes for f32, add in ((False, False), (True, False), (True, True))]
    assert max(taken) <= bound and sum(t > 0 for t in taken) > len(sizes) // 4
    M, N, K = 504, 5120, 65536                             # 40 tiles: 7 parts of each would be 73 MB
    a, b = (torch.randn(n, K, device="cuda").bfloat16() for n in (M, N))
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    e.gemm_bf16_2cta(a, b, out, False, True, False)
    want = a.double() @ b.double().t()
    # one rounding to bfloat16 of sums of K products in 32 bits
    assert (out.double() - want).abs().max() <= 2.0 ** -8 * want.abs().max() + 2.0 ** -20 * K
