"""The short convolution's register window: sequence starts inside and at the edges of a step and of a row block, every
filter width, values that are not finite, against the torch formulation."""
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


@pytest.mark.gpu
@pytest.mark.parametrize("W", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_values_that_are_not_finite_stay_inside_the_window(W, value):
    """A gradient row that is not finite reaches the W rows up to it in its sequence, a tap that is not finite the rows that
    have one that far behind; no others, also for filters shorter than the unrolled four taps.  Small integers elsewhere, so
    sums are exact."""
    from torchturbo_b200.ops import ops

    T, D, cu = 14, 8, [0, 5, 6, 14]
    gen = torch.Generator().manual_seed(W)
    ints = lambda *s: torch.randint(1, 4, s, generator=gen).float()                                       # noqa: E731
    first = [max(a for a in cu if a <= t) for t in range(T)]
    x, w, dy = ints(T, D), ints(D, W), ints(T, D)
    dy[4, 1] = dy[9, 2] = dy[13, 3] = value
    far = ints(D, W)
    far[5, 0] = value                                            # the tap of the oldest row
    for weight in (w, far):
        y, dx = torch.zeros(T, D), torch.zeros(T, D)
        for t in range(T):
            for s in range(W):
                if t - s >= first[t]:
                    y[t] += weight[:, W - 1 - s] * x[t - s]
                    dx[t - s] += weight[:, W - 1 - s] * dy[t]
        leaf = x.to("cuda", torch.bfloat16).unsqueeze(0).requires_grad_(True)
        got, _ = ops.causal_conv1d(leaf, weight.to("cuda", torch.bfloat16), None, activation=None, cu_seqlens=torch.tensor(cu))
        got.backward(dy.to("cuda", torch.bfloat16).unsqueeze(0))
        for a, b in ((got[0], y), (leaf.grad[0], dx)):
            assert torch.equal(torch.nan_to_num(a.detach().float().cpu(), nan=-777.0), torch.nan_to_num(b, nan=-777.0))
