"""A loss's saved gradient times the loss's gradient: the kernel against the torch passes, bit for bit, and who takes it."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 7, 8, 9, 2047, 2049, 8 * 256 * 148 * 8 + 11])
@pytest.mark.parametrize("src", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("dst", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shift", [0, 1])
def test_scale(n, src, dst, shift):
    from torchturbo_b200 import kernels as K

    x = torch.randn(n + shift, device="cuda").to(src)[shift:]
    if n > 8:
        x[3], x[5] = float("inf"), float("nan")
    g = torch.tensor(0.0371, device="cuda")
    got = K.scale(x, g, dst)
    want = (x.float() * g).to(dst)
    assert got.dtype == dst and torch.equal(got.nan_to_num(7.0), want.nan_to_num(7.0)) and torch.equal(got.isnan(), want.isnan())


def test_refused():
    from torchturbo_b200 import kernels as K

    x = torch.randn(8, 8, device="cuda")
    for args in ((x.t(), x[0, :1], torch.float32), (x, x[0, :2], torch.float32), (x, x[0, :1].bfloat16(), torch.float32),
                 (x.double(), x[0, :1], torch.float32)):
        with pytest.raises(AssertionError):
            K.scale(*args)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_loss_gradients_as_by_torch_passes(dtype):
    """A scaled loss backward, the same inside a graph of the gradient, and batched gradients, which see torch operations."""
    from torchturbo_b200.ops import ops

    torch.manual_seed(0)
    x = torch.randn(9, 520, device="cuda").to(dtype).requires_grad_(True)
    labels = torch.randint(0, 520, (9,), device="cuda")
    loss = ops.cross_entropy_loss(x, labels)
    f = torch.tensor(0.37, device="cuda", requires_grad=True)
    (plain,) = torch.autograd.grad(loss, x, f.detach(), retain_graph=True)
    (graph,) = torch.autograd.grad(loss, x, f, create_graph=True, retain_graph=True)
    assert torch.equal(plain, graph.detach()) and graph.requires_grad
    (back,) = torch.autograd.grad(graph.float().sum(), f, retain_graph=True)
    assert back.isfinite()
    (batch,) = torch.autograd.grad(loss, x, torch.stack((f.detach(), f.detach() * 2)), is_grads_batched=True)
    assert torch.equal(batch[0], plain) and batch.shape == (2, 9, 520)
