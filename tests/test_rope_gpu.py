"""The rotary kernel against the torch formulation, forward and backward, over strides and odd sizes."""
import pytest
import torch

from torchturbo_b200.ops import ops
from torchturbo_b200.ops.providers.native import rope_ref


@pytest.mark.gpu
@pytest.mark.parametrize("T, heads, D, layout", [
    (1, 1, 8, "plain"), (37, 16, 72, "qkv"), (64, 3, 64, "slice"), (129, 2, 128, "odd"), (300, 1, 24, "expand"), (33, 2, 12, "plain")])
def test_rope_kernel_matches_the_torch_formulation(T, heads, D, layout):
    """fp32 arithmetic and one rounding on both sides: equal up to the last bf16 bit (contraction of the products)."""
    torch.manual_seed(T)
    if layout == "qkv":
        x0 = torch.randn(T, 3, heads, D, device="cuda").to(torch.bfloat16)[:, 1]
    elif layout == "slice":
        x0 = torch.randn(T, heads, D + 128, device="cuda").to(torch.bfloat16)[..., 128:]
    elif layout == "odd":                                 # rows that start on a 2-byte boundary are copied first
        x0 = torch.randn(T * heads * D + 1, device="cuda").to(torch.bfloat16)[1:].view(T, heads, D)
    elif layout == "expand":
        x0 = torch.randn(T, 1, D, device="cuda").to(torch.bfloat16).expand(T, 4, D)
    else:
        x0 = torch.randn(T, heads, D, device="cuda").to(torch.bfloat16)
    ang = torch.randn(T, D // 2, device="cuda") * 10
    outs = []
    for fn in (ops.rotary_position_embedding, rope_ref):
        x = x0.detach().requires_grad_(True)
        y = fn(x, ang.cos(), ang.sin())
        y.backward(torch.cos(torch.arange(y.numel(), device="cuda").float()).view(y.shape).to(torch.bfloat16))
        outs.append((y.detach(), x.grad))
    for a, b in zip(*outs):
        assert a.shape == b.shape and a.dtype == b.dtype
        assert (a.float() - b.float()).abs().max() <= 2 ** -8 * b.float().abs().max()
        assert (a.float() - b.float()).norm() <= 2 ** -9 * b.float().norm()
