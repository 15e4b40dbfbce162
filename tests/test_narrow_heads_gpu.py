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


def _layouts(T, H, D):
    """Tensors that count as contiguous, or need no copy of their own, but whose strides are not those of dense rows."""
    rnd = lambda *s: torch.randn(*s, device="cuda").bfloat16()                                       # noqa: E731
    flat = rnd(T * H * D + 64)
    return {
        "one head, its stride that of all rows": rnd(1, T, D).transpose(0, 1) if H == 1 else None,
        "one token, an odd stride between rows": flat.as_strided((T, H, D), (H * D + 3, D, 1)) if T == 1 else None,
        "one token for the kernels to repeat": rnd(H, D).expand(T, H, D),
        "channels apart": rnd(T, H, 2 * D)[..., ::2],
        "heads first": rnd(H, T, D).transpose(0, 1),
        "overlapping rows": flat.as_strided((T, H, D), (8, D, 1)) if T <= 8 else None,
    }


@pytest.mark.parametrize("T,H,D", [(50, 1, 64), (1, 1, 72), (1, 3, 64), (7, 2, 40), (130, 2, 72)])
def test_layouts(T, H, D):
    """What has a layout of its own is taken, and gives what dense rows give."""
    cu = torch.tensor([0, T], dtype=torch.int32)
    dense = torch.randn(T, H, D, device="cuda").bfloat16()
    do = torch.randn(T, H, D, device="cuda").bfloat16()
    for name, t in _layouts(T, H, D).items():
        if t is None:
            continue
        for place in range(3):
            args = [dense, dense.flip(0), dense.neg()]
            args[place] = t
            got, ref = (_run(*(x.clone(memory_format=torch.contiguous_format) if dense_rows else x for x in args), cu, True, do, False)
                        for dense_rows in (False, True))
            for a, b in zip(got, ref):
                # one or two key blocks: the sums of at most two terms come out the same in either order
                assert torch.equal(a, b), (name, place)


def test_rows_of_heads():
    """The check itself, without a kernel: strides decide, not `is_contiguous`."""
    for T, H, D in ((50, 1, 64), (1, 3, 64), (1, 1, 8), (7, 2, 40)):
        for name, t in _layouts(T, H, D).items():
            if t is not None:
                r = A._rows_of_heads(t)
                assert torch.equal(r, t) and r.stride()[1:] == (D, 1) and r.stride(0) >= H * D and r.stride(0) % 8 == 0, name
    wide = torch.randn(9, 4, 64, device="cuda").bfloat16()
    assert A._rows_of_heads(wide[:, 1:3]).data_ptr() == wide[:, 1:3].data_ptr()                      # rows further apart stay where they are


def test_no_columns():
    """Heads without columns have uniform weights, or no result: they keep the padded way."""
    q, v = torch.zeros(20, 1, 0, device="cuda", dtype=torch.bfloat16), torch.randn(20, 1, 64, device="cuda").bfloat16()
    cu = torch.tensor([0, 20], dtype=torch.int32)
    o = ops.attention(q, q, v, cu, causal=False, scale=1.0)
    assert float((o.float() - v.float().mean(0)).abs().max()) < 2.0 ** -8
    assert ops.attention(v, v, v[..., :0], cu, causal=False).shape == (20, 1, 0)


def test_widths_that_are_no_multiple_of_eight_are_padded():
    q = torch.randn(50, 2, 20, device="cuda").bfloat16()
    assert not A._narrow(q, q, q) and A._paddable(q, q, q)
    o = ops.attention(q, q, q, torch.tensor([0, 50], dtype=torch.int32), causal=True)
    assert o.shape == q.shape and bool(torch.isfinite(o.float()).all())
