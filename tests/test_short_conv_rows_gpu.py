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
    """y, dw and db are fp32 sums rounded to bf16 once: half a unit in the last place is 2^-8 of the value, with sums in another order
    and fast exponentials 1e-5 of the magnitudes more.  The rows of dpre are rounded to bf16 before up to W of them meet in dx: 2^-8
    of their magnitudes besides."""
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
    # magnitudes: what the absolute values of all terms add up to
    xf, wf, bf, dyf = (t.float() for t in (x, w, b, dy))
    pre = causal_conv1d_ref(xf, wf, bf, None, None, False, cu)[0].requires_grad_(True)
    dpre = torch.autograd.grad(torch.nn.functional.silu(pre), pre, dyf)[0] if silu else dyf
    terms = [t.abs().requires_grad_(True) for t in (xf, wf, bf)]
    mag_y = causal_conv1d_ref(*terms, None, None, False, cu)[0]
    mags = [mag_y.detach(), *torch.autograd.grad(mag_y, terms, dpre.abs())]
    for name, a, ref, mag in zip(("y", "dx", "dw", "db"), *res, mags):
        a, ref = a.detach().float(), ref.detach().float()
        bound = 2.0 ** -8 * (ref.abs() + (mag if name == "dx" else 0)) + 1e-5 * mag + 1e-6
        assert bool(((a - ref).abs() <= bound).all()), (name, float(((a - ref).abs() - bound).max()))
        assert (a - ref).norm() <= 2 ** -8 * ref.norm() + 1e-6, ((a - ref).norm() / ref.norm())
