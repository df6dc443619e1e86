"""Autograd nodes in C++ against the Functions in Python that they stand in for: the same outputs, gradients, saved tensors and side effects."""
import pytest
import torch
from torch.utils.checkpoint import checkpoint

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _rand(*shape, dtype=BF16, seed=0, grad=True):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, generator=g, device="cuda").to(dtype).requires_grad_(grad)


def _cases():
    from neuronx_distributed_b200 import ops
    from neuronx_distributed_b200.parallel_layers.layers import tp_linear
    from neuronx_distributed_b200.parallel_layers.loss_functions import parallel_cross_entropy

    cos, sin = ops.rope.rope_tables(64, 128, device="cuda")
    target = (torch.arange(128, device="cuda") * 37 % 1000).view(64, 2)
    strided = lambda *s: _rand(s[1], s[0], *s[2:]).detach().transpose(0, 1).requires_grad_(True)
    return {
        "rms_norm": (lambda x, w: ops.norm.rms_norm(x, w, 1e-5), [_rand(64, 2, 512), _rand(512, seed=1)]),
        "rms_norm_strided": (lambda x, w: ops.norm.rms_norm(x, w, 1e-5), [strided(64, 2, 512), _rand(512, seed=1)]),
        "add_rms_norm": (lambda x, r, w: ops.norm.add_rms_norm(x, r, w, 1e-5), [_rand(64, 2, 512), _rand(64, 2, 512, seed=1), _rand(512, seed=2)]),
        "swiglu": (ops.act.swiglu, [_rand(64, 2, 512)]),
        "swiglu_f32": (ops.act.swiglu, [_rand(3, 32, dtype=torch.float32)]),
        "rope_qkv": (lambda x: ops.rope.rotary_qkv(x, cos, sin, 4, 2), [_rand(64, 2, 8 * 128)]),
        "attention": (lambda q, k, v: ops.attention.flash_attention(q, k, v), [_rand(2, 64, 4, 128), _rand(2, 64, 2, 128, seed=1), strided(2, 64, 2, 128)]),
        "loss": (lambda x: parallel_cross_entropy(x, target), [_rand(64, 2, 1000)]),
        "linear": (lambda x, w: tp_linear(x, w, None, "none", "none"), [_rand(256, 2, 256), _rand(512, 256, seed=1)]),
        "linear_few": (lambda x, w: tp_linear(x, w, None, "none", "none"), [_rand(24, 2, 256), _rand(64, 256, seed=1)]),
        "linear_8": (lambda x, w: tp_linear(x, w, None, "none", "none"), [_rand(8, 1, 256), _rand(512, 256, seed=1)]),
        "linear_odd": (lambda x, w: tp_linear(x, w, None, "none", "none"), [_rand(45, 1, 256), _rand(512, 256, seed=1)]),
        "linear_no_x": (lambda x, w: tp_linear(x, w, None, "none", "none"), [_rand(64, 2, 256, grad=False), _rand(512, 256, seed=1)]),
        "linear_no_w": (lambda x, w: tp_linear(x, w, None, "none", "none"), [_rand(64, 2, 256), _rand(512, 256, seed=1, grad=False)]),
    }


NAMES = ["rms_norm", "rms_norm_strided", "add_rms_norm", "swiglu", "swiglu_f32", "rope_qkv", "attention", "loss", "linear", "linear_few", "linear_8",
         "linear_odd", "linear_no_x", "linear_no_w"]


@pytest.fixture
def groups():
    import torch.distributed as dist
    from neuronx_distributed_b200.parallel_layers import parallel_state as ps

    if not dist.is_initialized():
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1, device_id=torch.device("cuda", 0))
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(tensor_model_parallel_size=1)


def _run(name, monkeypatch, native, how):
    from neuronx_distributed_b200.ops import _ext

    with monkeypatch.context() as m:
        if not native:
            m.setattr(_ext, "native", lambda *t: None)
        f, ins = _cases()[name]
        packed = []

        def pack(t):
            packed.append((tuple(t.shape), t.dtype))
            return t

        count = _ext.launches()
        if how == "checkpoint":
            out = checkpoint(f, *ins, use_reentrant=False)
        else:
            with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
                out = f(*ins)
        outs = out if isinstance(out, tuple) else (out,)
        gos = [_rand(*o.shape, dtype=o.dtype, seed=7 + i, grad=False) for i, o in enumerate(outs)]
        if how == "strided":
            gos = [g.repeat_interleave(2, -1)[..., ::2] for g in gos]
        need = [t for t in ins if t.requires_grad]
        first = outs if how != "one" else outs[:1]
        grads = torch.autograd.grad(first, need, gos[:len(first)], retain_graph=True, create_graph=how == "create", allow_unused=True)
        again = torch.autograd.grad(first, need, gos[:len(first)], allow_unused=True)
        return [o.detach() for o in outs], grads, again, packed, _ext.launches() - count, [(o.shape, o.stride(), o.dtype) for o in outs]


@pytest.mark.parametrize("how", ["plain", "one", "strided", "create", "checkpoint"])
@pytest.mark.parametrize("name", NAMES)
def test_native_node_is_the_function(name, how, groups, monkeypatch):
    a, b = (_run(name, monkeypatch, native, how) for native in (True, False))
    assert a[3:] == b[3:]                                  # what was saved, launches counted, shapes and strides
    for x, y in zip([*a[0], *a[1], *a[2]], [*b[0], *b[1], *b[2]]):
        assert (x is None) == (y is None)
        if x is not None:
            assert x.requires_grad == y.requires_grad and x.shape == y.shape and x.dtype == y.dtype
            if name == "attention":                        # sums over K/V tiles arrive in any order: fp32, then one rounding to bf16
                assert (x.double() - y.double()).abs().max() <= 2.0 ** -7 * y.double().abs().max()
            else:
                assert torch.equal(x, y)


@pytest.mark.parametrize("native", [True, False])
def test_weight_gradient_goes_into_its_buffer(native, groups, monkeypatch):
    from neuronx_distributed_b200.ops import _ext
    from neuronx_distributed_b200.parallel_layers.layers import tp_linear

    if not native:
        monkeypatch.setattr(_ext, "native", lambda *t: None)
    x, w = _rand(256, 1, 256), torch.nn.Parameter(_rand(512, 256, seed=1, grad=False))
    go = _rand(256, 1, 512, seed=3, grad=False)
    called = []
    want = go[:, 0].double().t() @ x.detach()[:, 0].double()
    for off in (0, 1):                                     # also a buffer that is not 16-byte aligned
        w.main_grad = torch.full((512 * 256 + 1,), 3.0, device="cuda")[off:off + 512 * 256].view(512, 256)
        w.main_grad_fresh, w._nxd_grad_ready = True, called.append
        for times in (1, 2):
            tp_linear(x, w, None, "none", "none").backward(go)
            assert w.grad is None and w.main_grad_fresh is False and called[-1] is w
            # fp32 sums of 256 exact products per element, added once or twice
            bound = 256 * 2.0 ** -23 * times * float((go[:, 0].abs().double().t() @ x.detach()[:, 0].abs().double()).max())
            assert (w.main_grad.double() - times * want).abs().max() <= bound
    monkeypatch.setenv("NXD_DISABLE_FUSED_WGRAD", "1")     # read by the backward pass
    before = w.main_grad.clone()
    tp_linear(x, w, None, "none", "none").backward(go)
    assert torch.equal(w.main_grad, before) and (w.grad.double() - want).norm() <= 2.0 ** -8 * want.norm()
    assert len(called) == 4


def test_nodes_in_python_where_the_others_cannot_go(groups):
    from torch.autograd import forward_ad

    from neuronx_distributed_b200 import ops

    x, w = _rand(16, 512, grad=False), _rand(512, seed=1, grad=False)
    with forward_ad.dual_level():
        assert ops._ext.native(x, w) is None
    assert ops._ext.native(x.cpu(), w) is None and ops._ext.native(x, w) is not None
    seen = []
    torch.func.vmap(lambda t: (seen.append(ops._ext.native(x)), t)[1])(x)
    assert seen == [None]

    class Sub(torch.Tensor):
        pass

    assert ops._ext.native(x.as_subclass(Sub)) is None
    with torch.inference_mode():
        y = ops.norm.rms_norm(x, w, 1e-5)
    assert torch.equal(y, ops.norm.rms_norm(x, w, 1e-5))
