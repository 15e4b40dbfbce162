"""The short convolution's register window: sequence starts inside and at the edges of a step and of a row block, every
filter width, against the torch formulation."""
import pytest
import torch

from torchturbo_b200.ops.providers.native_linear_attention import causal_conv1d_ref


@pytest.mark.gpu
@pytest.mark.parametrize("T, D, cu", [
    (1, 8, [0, 1]), (2, 16, [0, 1, 2]), (3, 8, [0, 3]), (5, 8, [0, 4, 5]), (37, 1032, [0, 1, 2, 3, 9, 37]),
    (300, 64, [0, 28, 29, 30, 57, 300]), (600, 2048, [0, 599, 600]), (1500, 8, [0, 700, 1500])])
@pytest.mark.parametrize("W", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("silu, with_bias", [(True, True), (False, False)])
def test_windows_stop_at_sequence_starts(T, D, cu, W, silu, with_bias):
    """bf16 results of fp32 sums of at most five products: 2^-8 of the largest value; dw and db are fp32 sums over T rows of
    terms that differ by bf16 roundings: 2^-7 of their norm."""
    from torchturbo_b200.ops import ops

    gen = torch.Generator().manual_seed(T * 8 + W)
    x = torch.randn(1, T, D, generator=gen).to(torch.bfloat16)
    w = torch.randn(D, W, generator=gen).to(torch.bfloat16)
    b = torch.randn(D, generator=gen).to(torch.bfloat16) if with_bias else None
    dy = torch.randn(1, T, D, generator=gen).to(torch.bfloat16)
    res = []
    for dev, dt in (("cuda", torch.bfloat16), ("cpu", torch.float32)):
        leaves = [t.to(dev, dt).requires_grad_(True) if t is not None else None for t in (x, w, b)]
        if dev == "cuda":
            y, _ = ops.causal_conv1d(*leaves, activation="silu" if silu else None, cu_seqlens=torch.tensor(cu))
        else:
            y, _ = causal_conv1d_ref(*leaves, "silu" if silu else None, None, False, cu)
        y.backward(dy.to(dev, dt))
        res.append([y] + [t.grad for t in leaves if t is not None])
    for a, b2 in zip(*res):
        a, b2 = a.detach().float().cpu(), b2.detach().float()
        assert (a - b2).norm() <= 2 ** -7 * b2.norm() + 1e-6, ((a - b2).norm() / b2.norm())
        assert (a - b2).abs().max() <= 2 ** -6 * max(1.0, b2.abs().max())
