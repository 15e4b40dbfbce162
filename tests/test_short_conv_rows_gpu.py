"""The short convolution over row blocks long enough for steps in which every tap of every row counts, against the torch formulation."""
import pytest
import torch

from torchturbo_b200.ops.providers.native_linear_attention import causal_conv1d_ref


@pytest.mark.gpu
@pytest.mark.parametrize("T, D, cu", [
    (1184, 4096, [0, 1184]), (1500, 8192, [0, 1, 3, 6, 10, 15, 21, 700, 707, 1499, 1500]), (2047, 8200, [0, 1000, 1020, 2047])])
@pytest.mark.parametrize("W", [3, 4])
@pytest.mark.parametrize("silu", [True, False])
def test_rows_inside_a_sequence(T, D, cu, W, silu):
    """bf16 results of fp32 sums of at most five products: 2^-8 of the largest value; dw and db are fp32 sums over T rows of
    terms that differ by bf16 roundings: 2^-7 of their norm."""
    from torchturbo_b200.ops import ops

    gen = torch.Generator("cuda").manual_seed(T + W)
    x, dy = (torch.randn(1, T, D, generator=gen, device="cuda").bfloat16() for _ in range(2))
    w, b = (torch.randn(D, *s, generator=gen, device="cuda").bfloat16() for s in ([W], []))
    res = []
    for dt in (torch.bfloat16, torch.float32):
        leaves = [t.to(dt).detach().requires_grad_(True) for t in (x, w, b)]
        if dt == torch.bfloat16:
            y, _ = ops.causal_conv1d(*leaves, activation="silu" if silu else None, cu_seqlens=torch.tensor(cu))
        else:
            y, _ = causal_conv1d_ref(*leaves, "silu" if silu else None, None, False, cu)
        y.backward(dy.to(dt))
        res.append([y] + [t.grad for t in leaves])
    for a, ref in zip(*res):
        a, ref = a.detach().float(), ref.detach().float()
        assert (a - ref).norm() <= 2 ** -7 * ref.norm() + 1e-6, ((a - ref).norm() / ref.norm())
        assert (a - ref).abs().max() <= 2 ** -6 * max(1.0, ref.abs().max())
