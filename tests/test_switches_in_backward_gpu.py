"""Switches of the environment that the backward pass reads, from autograd's own threads: late ones count, captured calls take them, and threads
that write os.environ meanwhile do no harm."""
import os
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _qkv(seed, seq=700, heads=4):
    g = torch.Generator(device="cuda").manual_seed(seed)
    q, k, v = (torch.randn(2, seq, h, 128, generator=g, device="cuda").bfloat16().requires_grad_() for h in (heads, 2, 2))
    return q, k, v, torch.randn(2, seq, heads, 128, generator=g, device="cuda").bfloat16()


def test_order_of_sums_asked_for_late_and_in_a_graph(monkeypatch):
    from neuronx_distributed_b200 import ops

    q, k, v, go = _qkv(0)
    o = ops.attention.flash_attention(q, k, v)
    monkeypatch.setenv("NXD_FA_DETERMINISTIC", "1")        # read by the backward pass
    want = [t.clone() for t in torch.autograd.grad(o, (q, k, v), go, retain_graph=True)]
    for _ in range(5):
        assert all(torch.equal(a, b) for a, b in zip(torch.autograd.grad(o, (q, k, v), go, retain_graph=True), want))
    graph = torch.cuda.CUDAGraph()                         # larger than any call before: its counters cannot be there yet
    q, k, v, go = _qkv(1, seq=900, heads=8)
    with torch.cuda.graph(graph):
        got = torch.autograd.grad(ops.attention.flash_attention(q, k, v), (q, k, v), go)
    graph.replay()
    want = torch.autograd.grad(ops.attention.flash_attention(q, k, v), (q, k, v), go)
    assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_backward_beside_writers_of_the_environment():
    from neuronx_distributed_b200 import ops

    def grads(seed):
        x, w = (t.requires_grad_() for t in _operands(seed))
        y = ops.act.swiglu(ops.norm.rms_norm(x, w, 1e-5))
        return torch.autograd.grad(y.float().square().sum(), (x, w))

    def _operands(seed):
        g = torch.Generator(device="cuda").manual_seed(seed)
        return torch.randn(300, 512, generator=g, device="cuda").bfloat16(), torch.randn(512, generator=g, device="cuda").bfloat16()

    want = [grads(s) for s in range(2)]
    bad, stop = [], threading.Event()

    def write():
        n = 0
        while not stop.is_set():
            n += 1
            os.environ[f"NXD_TEST_VALUE_{n % 50}"] = "x" * (n % 200)
            if n % 50 == 0:
                for i in range(50):
                    os.environ.pop(f"NXD_TEST_VALUE_{i}", None)

    def work(s):
        q, k, v, go = _qkv(s, seq=130)
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(60):
                if not all(torch.equal(a, b) for a, b in zip(grads(s), want[s])):
                    bad.append(s)
                torch.autograd.grad(ops.attention.flash_attention(q, k, v), (q, k, v), go)
        torch.cuda.synchronize()

    threads = [threading.Thread(target=write)] + [threading.Thread(target=work, args=(s,)) for s in range(2)]
    torch.cuda.synchronize()
    for t in threads:
        t.start()
    for t in threads[1:]:
        t.join()
    stop.set()
    threads[0].join()
    for i in range(50):
        os.environ.pop(f"NXD_TEST_VALUE_{i}", None)
    assert not bad
