"""The gate kernel of Kimi delta attention against its formula in 64 bits."""
import pytest
import torch

from torchturbo_b200.ops.providers.b200_linear_attention import KDAGate, _gate
from torchturbo_b200.ops.providers.native_linear_attention import kda_gate


@pytest.mark.gpu
@pytest.mark.parametrize("T, H", [(1, 1), (7, 3), (1200, 2), (33, 200)])
@pytest.mark.parametrize("bias, bound, dtype", [(True, None, torch.bfloat16), (False, None, torch.float32), (True, -5.0, torch.float32)])
def test_gate_and_its_gradients(T, H, bias, bound, dtype):
    """fp32 on one side, fp64 on the other; dg and bf16 parameter gradients add their rounding (2^-9)."""
    gen = torch.Generator().manual_seed(T)
    g0 = (torch.randn(1, T, H, 128, generator=gen) * 4).to(torch.bfloat16)
    g0[0, 0, 0, :3] = torch.tensor([30.0, -60.0, 20.5])              # linear branch, underflow, just behind the threshold
    A0 = torch.rand(H, generator=gen).mul(15).add(1).log().to(dtype)
    b0 = torch.randn(H * 128, generator=gen).to(dtype) if bias else None
    w = torch.randn(1, T, H, 128, generator=gen)
    leaves = [t.cuda().requires_grad_(True) if t is not None else None for t in (g0, A0, b0)]
    out = _gate(*leaves, bound)
    assert out.dtype == torch.float32 and out.grad_fn is not None
    (out * w.cuda()).sum().backward()
    ref = [t.double().requires_grad_(True) if t is not None else None for t in (g0, A0, b0)]
    x = ref[0] + (ref[2].view(H, 128) if bias else 0.0)
    a = ref[1].exp().view(H, 1)
    want = bound * torch.sigmoid(a * x) if bound is not None else -a * torch.nn.functional.softplus(x)
    (want * w.double()).sum().backward()
    assert (out.cpu().double() - want).abs().max() <= 4e-6 * want.abs().max()
    mine = kda_gate(g0.cuda(), A0.cuda(), b0.cuda() if bias else None, bound)
    assert (out - mine).abs().max() <= 4e-6 * mine.abs().max()
    for got, r, d in zip(leaves, ref, (torch.bfloat16, dtype, dtype)):
        if got is not None:
            tol = 2 ** -8 if d == torch.bfloat16 else 1e-5
            assert got.grad.dtype == got.dtype
            assert (got.grad.cpu().double() - r.grad).norm() <= tol * r.grad.norm() + 1e-7


@pytest.mark.gpu
def test_other_widths_take_the_formula():
    g = torch.randn(1, 5, 2, 64, device="cuda").to(torch.bfloat16)
    out = _gate(g, torch.zeros(2, device="cuda"), None, None)
    assert torch.equal(out, kda_gate(g, torch.zeros(2, device="cuda"), None, None)) and KDAGate is not None
