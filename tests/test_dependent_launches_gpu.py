"""Kernels that start beside their predecessor read what it wrote, weights too: chains in a stream and in a graph give what each step gives alone."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("rows,H,I", [(1, 4096, 1024), (2, 512, 4096), (4, 1024, 2816), (8, 4096, 4096), (48, 1024, 2816)])
def test_chain_reads_fresh_data(rows, H, I, graph):
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(rows)

    def rnd(*s):
        return torch.randn(*s, generator=g, device="cuda").bfloat16()

    src = [(rnd(rows, H), rnd(2 * I, H) * H ** -0.5, rnd(H, I) * I ** -0.5) for _ in range(3)]
    norm = rnd(H)
    x, w1, w2 = (torch.empty_like(t) for t in src[0])

    def chain(cur, stop):
        w1.copy_(cur[1])                                  # the weights themselves are written right before they are read
        x.copy_(cur[0])
        h = ops.norm.rms_norm(x, norm, 1e-5)
        stop()
        y = ops.gemm.matmul(h, w1, False, True)
        stop()
        a = ops.act.swiglu(y)
        stop()
        w2.copy_(cur[2])
        stop()
        z = ops.gemm.matmul(a, w2, False, True)
        stop()
        return ops.norm.rms_norm(z, norm, 1e-5)

    with torch.no_grad():
        want = [chain(cur, torch.cuda.synchronize).clone() for cur in src]
        go = lambda: None
        if graph:
            static = tuple(torch.empty_like(t) for t in src[0])
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                chain(static, go)
            torch.cuda.synchronize()
            program = torch.cuda.CUDAGraph()
            with torch.cuda.graph(program):
                out = chain(static, go)
        for i in range(60):
            if graph:
                for a, b in zip(static, src[i % 3]):
                    a.copy_(b)
                program.replay()
                got = out
            else:
                got = chain(src[i % 3], go)
            assert torch.equal(got, want[i % 3]), i
