"""Mean loss of a causal language model in the kernels' own launches, against the operations that it stands for and mathematics in 64 bits."""
import pytest
import torch
import torch.distributed as dist

pytestmark = pytest.mark.gpu


def _setup():
    from neuronx_distributed_b200.parallel_layers import parallel_state as ps

    if not dist.is_initialized():
        dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1)
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(tensor_model_parallel_size=1)


def _plain(logits, labels, shift):
    tgt = labels.t()
    if shift:
        tgt = torch.cat([tgt[1:], torch.full_like(tgt[:1], -100)])
    mask = tgt != -100
    rows = torch.nn.functional.cross_entropy(logits.flatten(0, 1), torch.where(mask, tgt, 0).flatten(), reduction="none").view(tgt.shape)
    return (rows * mask).sum() / mask.sum().clamp(min=1)


# one row, all hidden (every label, or the only position by the shift), blocks of 256 and 1024 rows and their remainders
@pytest.mark.parametrize("S,B,V,hidden", [(1, 1, 8, 0.), (2, 1, 16, 0.), (5, 3, 1001, 1.), (257, 1, 1000, .3), (128, 8, 520, .3), (1025, 3, 64, .9)])
@pytest.mark.parametrize("shift", [True, False])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_mean_and_gradient(S, B, V, hidden, shift, dtype):
    from neuronx_distributed_b200.parallel_layers.loss_functions import causal_lm_loss

    _setup()
    g = torch.Generator(device="cuda").manual_seed(S + V)
    x = (2 * torch.randn(S, B, V, generator=g, device="cuda")).to(dtype).requires_grad_()
    labels = torch.randint(0, V, (S, B), generator=g, device="cuda")
    labels[torch.rand(S, B, generator=g, device="cuda") < hidden] = -100
    for at in (labels.t(), labels.t().contiguous()):                      # both orders of the labels in memory
        loss = causal_lm_loss(x, at, shift)
        assert loss.dim() == 0 and loss.dtype == torch.float32
        x64 = x.detach().double().requires_grad_()
        want = _plain(x64, at, shift)
        kept = at.clone()
        at.fill_(0)                                                       # the next batch's labels may take the buffer
        loss *= 3.                                                        # in place, as programs that scale a loss do
        got, = torch.autograd.grad(loss, x)
        at.copy_(kept)
        (3 * want).backward()
        assert got.dtype == dtype
        # a row's loss: the sums' error 2^-16 of test_loss_rows_gpu; the mean: one rounding each of its quotient and its threefold
        assert abs(float(loss) - 3 * float(want)) <= 3 * (2 ** -16 + 2 ** -22 * abs(float(want)))
        # the exponential 2^-16 of the normaliser, its quotient and products 2^-22, one rounding to dtype
        tol = 2 ** -15 + (2 ** -8 if dtype == torch.bfloat16 else 0)
        assert (got.double() - x64.grad).abs().max() <= tol * float(x64.grad.abs().max())


def test_masked_rows_keep_their_infinities():
    """0 * loss of a hidden row is NaN where the loss is not finite, as in the operations that the kernels stand for."""
    from neuronx_distributed_b200.parallel_layers.loss_functions import causal_lm_loss, parallel_cross_entropy

    _setup()
    for bad in (float("nan"), float("inf"), float("-inf")):
        for col in (0, 3):
            x = torch.randn(4, 1, 64, device="cuda")
            x[2, 0, col] = bad
            labels = torch.tensor([[1, 2, 3, -100]], device="cuda")
            tgt = torch.cat([labels.t()[1:], torch.full((1, 1), -100, device="cuda")])
            mask = tgt != -100
            want = (parallel_cross_entropy(x, torch.where(mask, tgt, 0)) * mask).sum() / mask.sum()
            torch.testing.assert_close(causal_lm_loss(x, labels), want, equal_nan=True, rtol=1e-6, atol=1e-6)


def test_not_taken_and_captured():
    from neuronx_distributed_b200.parallel_layers.loss_functions import causal_lm_loss

    _setup()
    x, labels = torch.randn(6, 2, 64, device="cuda"), torch.randint(0, 64, (2, 6), device="cuda")
    assert causal_lm_loss(x.cpu(), labels.cpu()) is None and causal_lm_loss(x, labels.int()) is None
    assert causal_lm_loss(x, labels[:, :5]) is None and causal_lm_loss(x.double(), labels) is None and causal_lm_loss(x[:0], labels[:, :0]) is None
    want = causal_lm_loss(x, labels)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = causal_lm_loss(x, labels)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)


def test_recorded_gradients_and_recomputation():
    from torch.utils.checkpoint import checkpoint

    from neuronx_distributed_b200.parallel_layers.loss_functions import causal_lm_loss

    _setup()
    x, labels = torch.randn(70, 3, 520, device="cuda").bfloat16().requires_grad_(), torch.randint(0, 520, (3, 70), device="cuda")
    want, = torch.autograd.grad(causal_lm_loss(x, labels), x)
    for loss in (causal_lm_loss(x, labels), checkpoint(causal_lm_loss, x, labels, use_reentrant=False)):
        got, = torch.autograd.grad(loss, x, create_graph=True)
        again, = torch.autograd.grad(loss, x)
        assert torch.equal(got, want) and torch.equal(again, want)
