"""The gate kernel of Kimi delta attention against its formula in 64 bits."""
import pytest
import torch

from torchturbo_b200.ops.providers.b200_linear_attention import KDAGate, _gate
from torchturbo_b200.ops.providers.native_linear_attention import kda_gate


def test_row_blocks_cover_every_row_and_none_of_no_rows():
    import ctypes as C

    from torchturbo_b200 import kernels as K

    if not K.is_built():
        pytest.skip("library not built")
    blocks = lambda rows, H: K.lib().ttb_kda_gate_row_blocks(C.c_longlong(rows), C.c_int(H))                     # noqa: E731
    assert blocks(0, 3) == 0 and blocks(5, 0) == 0
    assert blocks(1, 1) == 1 and blocks(2047, 8) == 147 and blocks(33, 200) == 6


@pytest.mark.gpu
@pytest.mark.parametrize("T, H", [(0, 2), (1, 1), (7, 3), (1200, 2), (33, 200)])
@pytest.mark.parametrize("bias, bound, dtype", [(True, None, torch.bfloat16), (False, None, torch.float32), (True, -5.0, torch.float32)])
def test_gate_and_its_gradients(T, H, bias, bound, dtype):
    """fp32 on one side, fp64 on the other; dg and bf16 parameter gradients add their rounding (2^-9)."""
    gen = torch.Generator().manual_seed(T)
    g0 = (torch.randn(1, T, H, 128, generator=gen) * 4).to(torch.bfloat16)
    if T:
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
    if T:
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


@pytest.mark.gpu
@pytest.mark.parametrize("bound", [None, -5.0])
def test_gate_values_are_as_accurate_as_fp32_torch(bound):
    """Every value and every bias gradient (one row: nothing is summed) against 64 bits: the largest relative error is at most
    twice that of the same formula in fp32 torch.  Approximate exponentials are off by |x| 2^-24, thirty times as much at -60."""
    H = 64
    gen = torch.Generator().manual_seed(0)
    g = (torch.rand(1, 1, H, 128, generator=gen) * 90 - 60).to(torch.bfloat16)
    A = (torch.rand(H, generator=gen) * 2 - 2).bfloat16().float()
    bias = torch.zeros(H * 128)
    if bound is not None:                                   # sigmoid(a x) with a x exact: only the exponential rounds
        A = torch.zeros(H)
    res = []
    for fn, dev, dt in ((_gate, "cuda", None), (kda_gate, "cuda", None), (None, "cpu", torch.float64)):
        leaves = [t.to(dev, dt) if dt else t.to(dev) for t in (g, A, bias)]
        leaves[2].requires_grad_(True)
        if fn is not None:
            out = fn(*leaves, bound)
        else:
            x, a = leaves[0] + leaves[2].view(H, 128), leaves[1].exp().view(H, 1)
            out = bound * torch.sigmoid(a * x) if bound is not None else -a * torch.nn.functional.softplus(x)
        out.sum().backward()
        res.append([out.detach().double().cpu().reshape(-1), leaves[2].grad.double().cpu()])
    for mine, fp32, want in zip(*res):
        big = want.abs() > 2 ** -120
        err, ref = (((t - want).abs() / want.abs())[big].max().item() for t in (mine, fp32))
        assert err <= 2 * ref + 2 ** -23, (err, ref)


@pytest.mark.gpu
def test_bound_given_as_a_tensor_takes_the_formula():
    g, A, bound = torch.randn(1, 5, 2, 128, device="cuda").to(torch.bfloat16), torch.zeros(2, device="cuda"), torch.tensor(-5.0, device="cuda")
    assert torch.equal(_gate(g, A, None, bound), kda_gate(g, A, None, bound))
