"""QK-norm + RoPE over odd token and head counts, padded and misaligned rows, against the torch formulation."""
import pytest
import torch

from torchturbo_b200.ops import ops
from torchturbo_b200.ops.providers import native as N


@pytest.mark.gpu
@pytest.mark.parametrize("T, n_q, n_kv, layout, norm", [(1, 1, 0, "plain", True), (1, 1, 1, "plain", True), (3, 2, 1, "padded", True),
                                                        (257, 5, 2, "odd", True), (65, 4, 1, "plain", False), (1000, 32, 4, "plain", True)])
def test_values_and_gradients(T, n_q, n_kv, layout, norm):
    """Both sides round after the norm, after the weight and at the end; sums run in another order: a few bf16 units."""
    torch.manual_seed(T)
    width = (n_q + 2 * n_kv) * 128
    if layout == "padded":
        x0 = torch.randn(T, width + 64, device="cuda").to(torch.bfloat16)[:, :width]
    elif layout == "odd":
        x0 = torch.randn(T * (width + 1) + 1, device="cuda").to(torch.bfloat16)[1:].view(T, width + 1)[:, :width]
    else:
        x0 = torch.randn(T, width, device="cuda").to(torch.bfloat16)
    ang = torch.randn(T, 64, device="cuda")
    w0 = [(1 + 0.1 * torch.randn(128, device="cuda")).to(torch.bfloat16) for _ in range(2)]
    outs = []
    for fn in (ops.qk_norm_rope, N.TorchQKNormRope()):
        x = x0.detach().requires_grad_(True)
        w = [t.detach().requires_grad_(True) if norm else None for t in w0]
        q, k, v = fn(x, n_q, n_kv, 128, w[0], w[1], ang.cos(), ang.sin(), 1e-6)
        loss = sum((t.float() * torch.sin(torch.arange(t.numel(), device="cuda")).view(t.shape)).sum() for t in (q, k, v))
        loss.backward()
        outs.append([q, k, v, x.grad] + ([w[0].grad, w[1].grad] if norm else []))
    for a, b in zip(*outs):
        if b is None or b.numel() == 0:
            continue
        a, b = a.float(), b.float()
        assert (a - b).norm() <= 2 ** -6 * b.norm() + 1e-6, ((a - b).norm() / b.norm())
