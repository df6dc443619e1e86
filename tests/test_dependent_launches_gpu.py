"""Kernels that start beside their predecessor read what it wrote, weights too: chains in a stream and in a graph give what each step gives alone.
Forward and backward from threads of their own: test_switches_in_backward_gpu.py."""
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


def _alternate(program, sources, graph, equal, times=40):
    """``program(inputs, stop)`` over sources in turn, in one stream or as a graph, against itself with a halt at each ``stop()``."""
    want = [[t.clone() for t in program(cur, torch.cuda.synchronize)] for cur in sources]
    torch.cuda.synchronize()
    if graph:
        static = [torch.empty_like(t) for t in sources[0]]
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for a, b in zip(static, sources[0]):
                a.copy_(b)
            program(static, lambda: None)
        torch.cuda.synchronize()
        captured = torch.cuda.CUDAGraph()
        with torch.cuda.graph(captured):
            out = program(static, lambda: None)
    for i in range(times):
        cur = sources[i % len(sources)]
        if graph:
            for a, b in zip(static, cur):
                a.copy_(b)
            captured.replay()
        else:
            out = program(cur, lambda: None)
        for j, (a, b) in enumerate(zip(out, want[i % len(sources)])):
            equal(a, b, (i, j))


def _same(a, b, where):
    assert torch.equal(a, b), where


def _close(a, b, where):
    # sums in any order: fp32, then roundings to bf16 on the way; other inputs' results are as far off as the results are large
    assert (a.double() - b.double()).norm() <= 2.0 ** -6 * b.double().norm(), where


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("rows,H,I", [(200, 1024, 2816), (200, 8192, 3584), (1000, 5120, 6912)])      # the last two: a split tail
def test_many_rows_and_weights_that_a_norm_writes(rows, H, I, graph):
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(rows)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    gains = [torch.full((n,), n ** -0.5, device="cuda").bfloat16() for n in (H, I)]

    def program(cur, stop):
        x, r, w1, w2 = cur
        h, _ = ops.norm.add_rms_norm(x, r, gains[0] * H ** 0.5, 1e-5)
        stop()
        w = ops.norm.rms_norm(w1, gains[0], 1e-5)          # the weight comes from the launch right before the product
        stop()
        y = ops.gemm.matmul(h, w, False, True)
        stop()
        a = ops.act.swiglu(y)
        stop()
        w = ops.norm.rms_norm(w2, gains[1], 1e-5)
        stop()
        z = ops.gemm.matmul(a, w, False, True)
        stop()
        back = ops.gemm.matmul(z, w, False, False)         # as an input's gradient
        stop()
        grad = torch.full((H, I), 1.0, device="cuda")
        ops.gemm.matmul(z[:rows // 8 * 8], a[:rows // 8 * 8], True, False, out=grad, accumulate=True)
        stop()
        return [h, y, a, z, back, grad]

    with torch.no_grad():
        _alternate(program, [[rnd(rows, H), rnd(rows, H), rnd(2 * I, H), rnd(H, I)] for _ in range(2)], graph, _close if H * I > 1 << 24 else _same)


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("ordered", [False, True])
def test_training_block_both_ways(ordered, graph, monkeypatch):
    import torch.distributed as dist

    from neuronx_distributed_b200 import ops
    from neuronx_distributed_b200.parallel_layers import parallel_state as ps
    from neuronx_distributed_b200.parallel_layers.layers import tp_linear
    from neuronx_distributed_b200.parallel_layers.loss_functions import parallel_cross_entropy

    if not dist.is_initialized():
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1, device_id=torch.device("cuda", 0))
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(tensor_model_parallel_size=1)
    if ordered:
        monkeypatch.setenv("NXD_FA_DETERMINISTIC", "1")
        monkeypatch.setenv("NXD_GEMM_SPLITK", "0")
    S, B, heads, kv, V = 264, 2, 8, 2, 1000
    H, I = heads * 128, 1408
    g = torch.Generator(device="cuda").manual_seed(0)
    rnd = lambda *s, scale=1.0: (scale * torch.randn(*s, generator=g, device="cuda")).bfloat16()
    cos, sin = ops.rope.rope_tables(S, 128, device="cuda")
    target = (torch.arange(S * B, device="cuda") * 37 % V).view(S, B)
    linear = lambda x, w: tp_linear(x, w, None, "none", "none")

    def program(cur, stop):
        def seen(t):
            stop()
            if t.requires_grad:
                t.register_hook(lambda grad: stop())
            return t

        x, n1, wq, wo, n2, wg, wd, head = cur = [t.detach().requires_grad_() for t in cur]
        h = seen(ops.norm.rms_norm(x, n1, 1e-5))
        q, k, v = ops.rope.rotary_qkv(seen(linear(h, wq)), cos, sin, heads, kv)
        o = seen(ops.attention.flash_attention(seen(q), seen(k), v))
        o = seen(linear(o.transpose(0, 1).reshape(S, B, H), wo))
        y, r = ops.norm.add_rms_norm(o, x, n2, 1e-5)
        y = seen(linear(seen(ops.act.swiglu(seen(linear(seen(y), wg)))), wd))
        loss = seen(parallel_cross_entropy(seen(linear(y + r, head)), target))
        return [loss.detach(), *torch.autograd.grad(loss.mean(), cur)]

    def source():
        return [rnd(S, B, H), 1 + rnd(H, scale=0.1), rnd((heads + 2 * kv) * 128, H, scale=H ** -0.5), rnd(H, H, scale=H ** -0.5), 1 + rnd(H, scale=0.1),
                rnd(2 * I, H, scale=H ** -0.5), rnd(H, I, scale=I ** -0.5), rnd(V, H, scale=H ** -0.5)]

    _alternate(program, [source() for _ in range(2)], graph, _same if ordered else _close)


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("B,heads,kv,longest", [(1, 8, 8, 300), (3, 8, 2, 2000)])
def test_token_chain(B, heads, kv, longest, graph):
    from neuronx_distributed_b200 import ops

    e, H = ops._ext.ext(), heads * 128
    g = torch.Generator(device="cuda").manual_seed(longest)
    rnd = lambda *s, scale=1.0: (scale * torch.randn(*s, generator=g, device="cuda")).bfloat16()
    cos, sin = ops.rope.rope_tables(longest, 128, device="cuda")
    gain = torch.ones(H, device="cuda").bfloat16()

    def program(cur, stop):
        x, r, wq, wo, kc, vc, pos = cur
        kc, vc = kc.clone(), vc.clone()
        stop()
        h = ops.norm.rms_norm(x, gain, 1e-5)
        stop()
        qkv = ops.gemm.matmul(h, wq, False, True).view(B, 1, heads + 2 * kv, 128)
        stop()
        q, k, v = qkv.split([heads, kv, kv], 2)
        q = e.decode_rope_kv(q, k, v, pos, cos, sin, kc, vc)
        stop()
        o = ops.attention.decode_attention(q, kc, vc, pos).view(B, H)
        stop()
        w = ops.norm.rms_norm(wo, gain, 1e-5)              # the weight from the launch right before
        stop()
        y, s = ops.norm.add_rms_norm(e.gemv(o, w, None), r, gain, 1e-5)
        stop()
        return [h, qkv, kc, vc, o, y, s]

    def source(i):
        pos = torch.tensor([(longest - 1 - 7 * (b + i)) % longest for b in range(B)], device="cuda")
        return [rnd(B, H), rnd(B, H), rnd((heads + 2 * kv) * 128, H, scale=H ** -0.5), rnd(H, H), rnd(B, longest, kv, 128), rnd(B, longest, kv, 128), pos]

    with torch.no_grad():
        _alternate(program, [source(i) for i in range(3)], graph, _same)


@pytest.mark.parametrize("graph", [False, True])
def test_two_streams_that_wait_for_one_another(graph):
    """A dependent launch behind an event waits for the other stream's work too, not only for the launch before it in its own."""
    from neuronx_distributed_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(5)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    gain, w = torch.ones(1024, device="cuda").bfloat16(), rnd(1024, 1024) * 0.03
    other = torch.cuda.Stream()

    def program(cur, stop):
        x, y = cur
        here = torch.cuda.current_stream()
        other.wait_stream(here)
        with torch.cuda.stream(other):
            torch.cuda._sleep(200000)                      # the other stream is late
            a = ops.norm.rms_norm(x, gain, 1e-5)
            a = ops.gemm.matmul(a, w, False, True)
        stop()
        b = ops.norm.rms_norm(y, gain, 1e-5)               # the launch before, done long ago
        stop()
        here.wait_stream(other)
        c, s = ops.norm.add_rms_norm(a, b, gain, 1e-5)
        stop()
        other.wait_stream(here)
        with torch.cuda.stream(other):
            d = ops.gemm.matmul(c, w, False, True)
        here.wait_stream(other)
        stop()
        for t in (a, d):
            t.record_stream(here)
        for t in (x, c):
            t.record_stream(other)
        return [b, c, s, ops.norm.rms_norm(d, gain, 1e-5)]

    with torch.no_grad():
        _alternate(program, [[rnd(300, 1024), rnd(300, 1024)] for _ in range(2)], graph, _same)
