"""The rotary kernel against the torch formulation: forward and backward over strides and odd sizes, higher derivatives, and
the transforms and tracers under which the operator stays made of torch operations."""
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


def _second(fn, x, probe):
    """d/dx of <grad of sum(fn(x)^2 + x^3), probe>."""
    x = x.detach().requires_grad_(True)
    y = fn(x)
    (g,) = torch.autograd.grad((y.float() ** 2).sum() + (x.float() ** 3).sum(), x, create_graph=True)
    (h,) = torch.autograd.grad((g.float() * probe).sum(), x)
    return g.detach().float(), h.float()


def test_gradient_of_the_gradient_goes_through_the_rotation(monkeypatch):
    """The autograd function around a stand-in for the kernel, which autograd cannot see through either."""
    from torchturbo_b200.ops.providers import b200

    def kernel(x, cos, sin, sign=1.0):
        with torch.no_grad():
            return rope_ref(x, cos, sign * sin)

    monkeypatch.setattr(b200.K, "rope", kernel)
    torch.manual_seed(0)
    x, ang, probe = torch.randn(5, 2, 16), torch.randn(5, 8), torch.randn(5, 2, 16)
    got = _second(lambda t: b200.RopeFn.apply(t, ang.cos(), ang.sin(), 1.0), x, probe)
    want = _second(lambda t: rope_ref(t, ang.cos(), ang.sin()), x, probe)
    for a, b in zip(got, want):
        assert torch.allclose(a, b, atol=1e-5, rtol=1e-5)


def test_only_ordinary_tensors_outside_transforms_are_eager():
    from torch.autograd import forward_ad
    from torch.fx.experimental.proxy_tensor import make_fx

    from torchturbo_b200.ops.providers.b200 import _eager

    x, seen = torch.randn(3, 4), []
    note = lambda t: seen.append(_eager(t)) or t.sin()                                                    # noqa: E731
    note(x)
    note(torch.nn.Parameter(x))
    torch.func.vmap(note)(x)
    torch.func.jvp(note, (x,), (x,))
    torch.func.grad(lambda t: note(t).sum())(x)
    make_fx(note)(x)
    torch.jit.trace(note, (x,), check_trace=False)
    with forward_ad.dual_level():
        note(forward_ad.make_dual(x, x))
        note(x)
    note(torch.Tensor._make_subclass(type("Sub", (torch.Tensor,), {}), x))
    assert seen == [True, True, False, False, False, False, False, False, True, False]


@pytest.mark.gpu
def test_second_derivative_and_transforms_match_the_torch_formulation():
    """bf16 gradients on both sides: 2^-7 of the largest entry (two roundings on the way to the second derivative)."""
    torch.manual_seed(1)
    x = torch.randn(33, 4, 64, device="cuda").to(torch.bfloat16)
    ang, probe = torch.randn(33, 32, device="cuda"), torch.randn(33, 4, 64, device="cuda")
    cos, sin = ang.cos(), ang.sin()
    op = lambda t: ops.rotary_position_embedding(t, cos, sin)                                             # noqa: E731
    ref = lambda t: rope_ref(t, cos, sin)                                                                 # noqa: E731
    for a, b in zip(_second(op, x, probe), _second(ref, x, probe)):
        assert (a - b).abs().max() <= 2 ** -7 * b.abs().max()
    batch = torch.stack((x, 2 * x))
    assert torch.equal(torch.func.vmap(op)(batch), torch.func.vmap(ref)(batch))
    for a, b in zip(torch.func.jvp(op, (x,), (x,)), torch.func.jvp(ref, (x,), (x,))):
        assert torch.equal(a, b)
