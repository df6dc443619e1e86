"""Product with [gate; up] weights and SwiGLU in one kernel, against mathematics in 64 bits and against the two kernels."""
import pytest
import torch

from neuronx_distributed_b200 import ops
from neuronx_distributed_b200.ops.gemm import _few_rows

pytestmark = pytest.mark.gpu


def _case(M, I, K):
    g = torch.Generator(device="cuda").manual_seed(M * 7 + I)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    w = torch.randn(2 * I, K, generator=g, device="cuda").mul_(K ** -0.5).bfloat16()
    return x, w


# rows for the vector kernel are left to it; few rows (tokens padded to 16, slabs of 64 + 64 rows of W, K split over clusters), CTA pairs (whole tiles, tails)
@pytest.mark.parametrize("M,I,K,taken", [(1, 2816, 1024, False), (2, 192, 72, False), (2, 11008, 4096, True), (3, 192, 72, False), (4, 3584, 8192, True),
                                         (8, 11008, 4096, True), (9, 64, 8, True), (16, 192, 1000, True), (48, 11008, 4096, True), (65, 2816, 1024, True),
                                         (128, 2816, 1024, True), (176, 11008, 4096, True), (200, 2816, 4096, True), (136, 2816, 1024, True), (256, 2816, 1024, True),
                                         (264, 128, 72, True), (1000, 13824, 5120, True), (520, 1408, 4096, True), (301, 2816, 1024, False), (264, 192, 72, False)])
def test_values(M, I, K, taken):
    x, w = _case(M, I, K)
    y = ops._ext.ext().linear_swiglu(x, w, _few_rows(M, 2 * I, K))
    assert (y is not None) == taken
    if not taken:
        return
    gate, up = (x.double() @ w.double().t()).chunk(2, -1)
    want = torch.nn.functional.silu(gate) * up
    # gate, up and the result are each rounded to bf16 once; silu's slope is at most 1.1
    assert float((y.double() - want).norm() / want.norm()) < 3.2 * 2 ** -9
    if M <= 8 or _few_rows(M, 2 * I, K):                    # the same sums: the same bits as two kernels give
        assert torch.equal(y, ops.act.swiglu(ops._ext.ext().gemv(x, w, None) if M <= 8 else ops._ext.ext().gemm_few_rows(x, w)))
    assert torch.equal(y, ops._ext.ext().linear_swiglu(x, w, _few_rows(M, 2 * I, K)))


def _mlp():
    import torch.distributed as dist

    from neuronx_distributed_b200.models.llama import LlamaConfig, LlamaMLP
    from neuronx_distributed_b200.parallel_layers import parallel_state as ps

    if not dist.is_initialized():
        dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1)
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(tensor_model_parallel_size=1)
    return LlamaMLP(LlamaConfig(hidden_size=256, intermediate_size=384, dtype=torch.bfloat16, device=torch.device("cuda", 0)))


def test_projections_that_somebody_watches_are_called():
    mlp, x = _mlp(), torch.randn(16, 1, 256, device="cuda").bfloat16()
    with torch.no_grad():
        plain = mlp(x)
        seen = []
        handle = mlp.gate_up_proj.register_forward_hook(lambda m, i, o: seen.append(o.shape))
        watched = mlp(x)
        handle.remove()
        handle = torch.nn.modules.module.register_module_forward_hook(lambda m, i, o: seen.append(type(m).__name__))
        mlp(x)
        handle.remove()
    assert seen[0] == (16, 1, 768) and "ColumnParallelLinear" in seen and torch.equal(plain, watched)
    assert mlp(x.requires_grad_()).requires_grad


# whole tiles, tails, a remainder of rows, several rows' dimensions; with and without a gradient of x, into the optimizer's buffer and as .grad
@pytest.mark.parametrize("shape,I", [((136, 1024), 2816), ((132, 2, 4096), 1408), ((1000, 72), 128), ((2, 260, 1024), 1408)])
@pytest.mark.parametrize("of_x,buffer", [(True, False), (False, False), (True, True)])
def test_gradients(shape, I, of_x, buffer):
    from neuronx_distributed_b200.parallel_layers.layers import ColumnParallelLinear, column_swiglu

    _mlp()
    K = shape[-1]
    x, w = _case(x_rows := torch.Size(shape[:-1]).numel(), I, K)
    x, go = x.view(shape), torch.randn(*shape[:-1], I, device="cuda").bfloat16()
    proj = ColumnParallelLinear(K, 2 * I, bias=False, gather_output=False, dtype=torch.bfloat16, device=torch.device("cuda", 0))
    proj.weight.data.copy_(w)

    def run(fused):
        proj.weight.grad = None
        if buffer:
            proj.weight.main_grad = torch.ones(2 * I, K, device="cuda")
            proj.weight.main_grad_fresh = False
        xi = x.clone().requires_grad_(of_x)
        before = ops._ext.launches()
        y = column_swiglu(proj, xi) if fused else ops.act.swiglu(proj(xi))
        launched = ops._ext.launches() - before
        y.backward(go)
        return y.detach(), xi.grad, proj.weight.main_grad if buffer else proj.weight.grad, launched

    one, two = run(True), run(False)
    assert (one[3], two[3]) == (1, 2) and x_rows > 128
    for a, b in zip(one[:3], two[:3]):
        assert (a is None) == (b is None)
        # the same products but for the order of a tail's sums, each rounded to bf16 on the way: 2^-9 of the gates and ups, silu's slopes at most 1.1
        assert a is None or float((a.double() - b.double()).norm() / b.double().norm()) < 2 ** -7
    gate, up = (x.double() @ w.double().t()).chunk(2, -1)
    want = torch.nn.functional.silu(gate) * up
    assert float((one[0].double() - want).norm() / want.norm()) < 3.2 * 2 ** -9
    handles = [proj.register_full_backward_hook(lambda m, gi, go: None)]
    before = ops._ext.launches()
    column_swiglu(proj, x.clone().requires_grad_(of_x))
    assert ops._ext.launches() - before == 2                 # a watched projection is called
    handles[0].remove()


def test_captured_graph_and_two_streams():
    x, w = _case(264, 1408, 1024)
    e = ops._ext.ext()
    want = e.linear_swiglu(x, w, False)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = e.linear_swiglu(x, w, False)
    y.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    got = []
    for i in range(8):
        with torch.cuda.stream(streams[i % 2]):
            got.append(e.linear_swiglu(x, w, False))
    torch.cuda.synchronize()
    assert all(torch.equal(t, want) for t in got)


@pytest.mark.parametrize("M", [9, 33, 63, 65, 127])
@pytest.mark.parametrize("grads", [False, True])
def test_rows_of_any_number(M, grads):
    """x Wᵀ of up to 64 rows runs on the few-row kernel whatever their number; more that are no multiple of 8 on the library's."""
    from neuronx_distributed_b200.parallel_layers.layers import tp_linear
    from neuronx_distributed_b200.parallel_layers import parallel_state as ps

    _mlp()
    x, w = _case(M, 192, 264)
    x.requires_grad_(grads), w.requires_grad_(grads)
    before = ops._ext.launches()
    with torch.set_grad_enabled(grads):
        y = tp_linear(x, w, None, "none", "none", group=ps.get_tensor_model_parallel_group())
    assert (ops._ext.launches() > before) == (M <= 64)
    want = x.double() @ w.double().t()
    assert float((y.double() - want).norm() / want.norm()) < 2 ** -8
    if grads:
        go = torch.randn_like(y)
        gx, gw = torch.autograd.grad(y, (x, w), go)
        for a, b in ((gx, go.double() @ w.double()), (gw, go.double().t() @ x.double())):
            assert float((a.double() - b).norm() / b.norm()) < 2 ** -8


def _peak_of_backward(forward, args):
    """Bytes above what is held before the backward pass."""
    y = forward()
    go = torch.ones_like(y)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    held = torch.cuda.memory_allocated()
    torch.autograd.grad(y, args, go)
    return torch.cuda.max_memory_allocated() - held


def test_products_are_given_back_before_the_gradients_are_computed():
    """The backward pass needs no more memory than that of the two nodes: gradients of 2 I columns, of x and of W without the products."""
    from neuronx_distributed_b200.parallel_layers.layers import ColumnParallelLinear, column_swiglu

    _mlp()
    M, I, K = 2048, 2816, 1024
    x, w = _case(M, I, K)
    proj = ColumnParallelLinear(K, 2 * I, bias=False, gather_output=False, dtype=torch.bfloat16, device=torch.device("cuda", 0))
    proj.weight.data.copy_(w)
    x.requires_grad_()
    one, two = (_peak_of_backward(f, (x, proj.weight)) for f in (lambda: column_swiglu(proj, x), lambda: ops.act.swiglu(proj(x))))
    assert one <= two + 2 ** 16 and one < 2 * (M * 2 * I + M * K + 2 * I * K)


def test_products_of_experts_are_given_back_before_the_gradients_are_computed():
    mb = ops.moe_blocks
    T, E, H, I = 2048, 4, 512, 1408
    idx = torch.stack([torch.randperm(E, device="cuda")[:2] for _ in range(T)])
    slots = mb.make_slots(idx, E, (2 * T + mb.BLOCK - 1) // mb.BLOCK + E)
    x = mb.gather(torch.randn(T, H, device="cuda").bfloat16(), slots).detach().requires_grad_()
    w = (torch.randn(E, H, 2 * I, device="cuda") * H ** -0.5).bfloat16().requires_grad_()
    a = (x, w, slots.block_expert, slots.seg, mb.BLOCK)
    one, two = (_peak_of_backward(f, (x, w)) for f in (
        lambda: ops.gemm.grouped_swiglu(*a, slots.token), lambda: ops.act.swiglu(ops.gemm.grouped_matmul(*a, skip_unused=True, slot_token=slots.token))))
    assert one <= two + 2 ** 16


# numbers of rows that are no multiple of 8 (and few or many of them): the two kernels or the library's, by the same rules as a plain projection
@pytest.mark.parametrize("M", [65, 97, 301, 777, 1001])
@pytest.mark.parametrize("grads", [False, True])
def test_rows_that_the_one_kernel_leaves(M, grads):
    mlp = _mlp()
    x, w = _case(M, 384, 256)
    mlp.gate_up_proj.weight.data.copy_(w)
    x, weights = x.view(M, 1, 256).requires_grad_(grads), (mlp.gate_up_proj.weight, mlp.down_proj.weight)
    with torch.set_grad_enabled(grads):
        y = mlp(x)
    ref = [t.detach().double().requires_grad_() for t in (x, *weights)]
    gate, up = (ref[0] @ ref[1].t()).chunk(2, -1)
    want = torch.nn.functional.silu(gate) * up @ ref[2].t()
    # gate, up, their SwiGLU and the result are each rounded to bf16 once; silu's slope is at most 1.1
    assert float((y.detach().double() - want).norm() / want.norm()) < 4.2 * 2 ** -9
    if grads:
        go = torch.randn_like(y)
        for a, b in zip(torch.autograd.grad(y, (x, *weights), go), torch.autograd.grad(want, ref, go.double())):
            assert float((a.double() - b).norm() / b.norm()) < 2 ** -6        # two more products, each of rounded factors


@pytest.mark.parametrize("how", ["create", "checkpoint", "hooks"])
def test_its_nodes_as_programs_use_them(how):
    """Recorded gradients, recomputation and hooks on what is saved: the results of a plain backward pass, and the same tensors saved."""
    from torch.utils.checkpoint import checkpoint

    from neuronx_distributed_b200.parallel_layers.layers import ColumnParallelLinear, column_swiglu

    _mlp()
    M, I, K = 264, 1408, 1024
    x, w = _case(M, I, K)
    proj = ColumnParallelLinear(K, 2 * I, bias=False, gather_output=False, dtype=torch.bfloat16, device=torch.device("cuda", 0))
    proj.weight.data.copy_(w)
    go = torch.randn(M, I, device="cuda").bfloat16()
    x.requires_grad_()
    want = torch.autograd.grad(column_swiglu(proj, x), (x, proj.weight), go)
    packed, before = [], ops._ext.launches()
    if how == "checkpoint":
        y = checkpoint(column_swiglu, proj, x, use_reentrant=False)
    elif how == "hooks":
        with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(tuple(t.shape)) or t.cpu(), lambda t: t.cuda()):
            y = column_swiglu(proj, x)
        assert sorted(packed) == sorted([(M, K), (2 * I, K), (M, 2 * I)])
    else:
        y = column_swiglu(proj, x)
    assert ops._ext.launches() - before == 1
    got = torch.autograd.grad(y, (x, proj.weight), go, retain_graph=True, create_graph=how == "create")
    again = torch.autograd.grad(y, (x, proj.weight), go)
    for a, b, c in zip(want, got, again):
        assert torch.equal(a, b) and torch.equal(a, c)
