"""Bias, split and rotary embedding between a fused projection and attention in one pass, against the operators it stands for."""
import pytest
import torch


def _same(a, b):
    """Both form x c - y s in fp32 (values up to 8), where the order of the two products is the compiler's: a unit of 2^-23 of them
    before the one rounding to bf16."""
    return ((a.float() - b.float()).abs() <= 2.0 ** -7 * b.float().abs() + 2.0 ** -20).all()


@pytest.mark.gpu
@pytest.mark.parametrize("T", [1, 37, 1200])
@pytest.mark.parametrize("heads, D", [(1, 8), (3, 40), (16, 72), (16, 88), (32, 128)])     # 3 to 1536 groups of four pairs a row
def test_same_results_as_the_separate_operators(T, heads, D):
    from torchturbo_b200.ops import ops
    from torchturbo_b200.ops.providers import native as N

    gen = torch.Generator("cuda").manual_seed(T + D)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen).bfloat16()      # noqa: E731
    ang = torch.rand(T, D // 2, device="cuda", generator=gen) * 6
    cos, sin = ang.cos(), ang.sin()
    res = []
    x0, b0, do = rnd(T, 3 * heads * D), rnd(3 * heads * D), [rnd(T, heads, D) for _ in range(3)]
    for op in (ops.qkv_bias_rope, N.TorchQKVBiasRope()):
        x, b = x0.clone().requires_grad_(), b0.clone().requires_grad_()
        out = op(x, b, heads, cos, sin)
        grads = torch.autograd.grad(out, (x, b), do)
        again = torch.autograd.grad(op(x, b, heads, cos, sin), (x, b), [t.clone().requires_grad_() for t in do], create_graph=True)
        assert _same(again[0], grads[0])
        res.append((out, grads))
    (out, (dx, db)), (want, (wx, wb)) = res
    assert torch.equal(out[2], want[2]) and all(_same(a, b) for a, b in zip((*out[:2], dx), (*want[:2], wx)))
    # sums of T values in another order (T units of 2^-24 of their magnitudes on either side), each rounded to bf16
    for got, terms in ((db, dx.double()), (wb, wx.double())):
        exact, mag = terms.sum(0), terms.abs().sum(0)
        assert ((got.double() - exact).abs() <= mag * T * 2.0 ** -24 + exact.abs() * 2.0 ** -8).all()


@pytest.mark.gpu
def test_a_choice_for_one_of_its_parts_is_kept():
    from torchturbo_b200.ops.ops import get_or_create_ops
    from torchturbo_b200 import kernels as K

    x, b = torch.randn(9, 48, device="cuda").bfloat16(), torch.randn(48, device="cuda").bfloat16()
    cos = sin = torch.ones(9, 4, device="cuda")
    ops = get_or_create_ops(overrides={"rotary_position_embedding": "native", "bias_act": "native"})
    try:
        n = K.launch_count()
        ops.qkv_bias_rope(x, b, 2, cos, sin)
        assert K.launch_count() == n
    finally:
        get_or_create_ops(reset=True)
