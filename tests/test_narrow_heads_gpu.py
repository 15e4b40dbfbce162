"""Attention heads narrower than 128 are taken as they are; the results are those of heads padded with zero columns."""
import pytest
import torch
import torch.nn.functional as F

from torchturbo_b200.ops import ops
from torchturbo_b200.ops.providers import b200_attention as A

pytestmark = pytest.mark.gpu


def _run(q, k, v, cu, causal, do, pad):
    D, Dv = q.shape[-1], v.shape[-1]
    q, k, v = (t.detach().requires_grad_(True) for t in (q, k, v))
    if pad:
        o = ops.attention(F.pad(q, (0, 128 - D)), F.pad(k, (0, 128 - D)), F.pad(v, (0, 128 - Dv)), cu, causal=causal, scale=D ** -0.5)[..., :Dv]
    else:
        o = ops.attention(q, k, v, cu, causal=causal)
    return (o.detach(), *torch.autograd.grad(o, (q, k, v), do))


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D,Dv,Hq,Hk", [(72, 72, 4, 4), (80, 80, 3, 3), (8, 16, 4, 2), (64, 128, 4, 1), (128, 40, 2, 2), (120, 96, 2, 1)])
def test_same_as_padded(D, Dv, Hq, Hk, causal, deterministic):
    cu = torch.tensor([0, 1, 130, 387, 515, 900], dtype=torch.int32)
    T = 910
    g = torch.Generator("cuda").manual_seed(D + Dv)
    q, k = (torch.randn(T, h, D, generator=g, device="cuda").bfloat16() for h in (Hq, Hk))
    v = torch.randn(T, 2 * Hk, Dv, generator=g, device="cuda").bfloat16()[:, Hk:]           # rows further apart than they are long
    do = torch.randn(T, Hq, Dv, generator=g, device="cuda").bfloat16()
    assert A._narrow(q, k, v)
    torch.use_deterministic_algorithms(deterministic, warn_only=True)
    try:
        got, ref = (_run(q, k, v, cu, causal, do, pad) for pad in (False, True))
    finally:
        torch.use_deterministic_algorithms(False)
    for a, b in zip(got, ref):
        assert a.shape == b.shape and bool(torch.isfinite(a.float()).all())
        # the same products in the same order; where fp32 sums of several blocks are added by atomics their order may differ, which
        # the rounding to bf16 turns into at most one unit in the last place here and there
        err = (a.float() - b.float()).abs()
        assert bool((err <= 2.0 ** -7 * b.float().abs() + 1e-5 * b.float().abs().max()).all())
        assert float((err > 0).float().mean()) < 0.05
        assert bool((a[900:] == 0).all())


@pytest.mark.parametrize("shift", [1, 4])
def test_operands_between_16_byte_boundaries(shift):
    T, H, D = 200, 2, 72
    flat = torch.randn(3 * T * H * D + 8, device="cuda").bfloat16()
    q, k, v = (flat[shift + i * T * H * D: shift + (i + 1) * T * H * D].view(T, H, D) for i in range(3))
    cu = torch.tensor([0, T], dtype=torch.int32)
    do = torch.randn(T * H * D + 8, device="cuda").bfloat16()[shift: shift + T * H * D].view(T, H, D)
    for a, b in zip(_run(q, k, v, cu, False, do, False), _run(q.clone(), k.clone(), v.clone(), cu, False, do.clone(), True)):
        assert float((a.float() - b.float()).abs().max()) <= 2.0 ** -7 * float(b.float().abs().max())


def test_widths_that_are_no_multiple_of_eight_are_padded():
    q = torch.randn(50, 2, 20, device="cuda").bfloat16()
    assert not A._narrow(q, q, q) and A._paddable(q, q, q)
    o = ops.attention(q, q, q, torch.tensor([0, 50], dtype=torch.int32), causal=True)
    assert o.shape == q.shape and bool(torch.isfinite(o.float()).all())
