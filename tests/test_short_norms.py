"""Gated RMSNorm of short rows and the column sums behind every norm's weight gradient."""
import pytest
import torch

from torchturbo_b200.ops import ops


@pytest.mark.parametrize("activation", ["silu", "sigmoid"])
def test_gated_norm_is_the_norm_times_the_activation_on_cpu(activation):
    torch.manual_seed(0)
    x, gate, w = torch.randn(7, 3, 16), torch.randn(7, 3, 16), torch.rand(16)
    got = ops.gated_rms_norm(x, gate, w, 1e-6, activation=activation, impl="torch_gated_rms_norm")
    act = torch.sigmoid(gate) * (gate if activation == "silu" else 1.0)
    want = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6) * w * act
    assert torch.allclose(got, want, atol=1e-6, rtol=1e-5)


@pytest.mark.parametrize("activation", ["silu", "sigmoid"])
def test_second_derivatives_go_through_the_separate_operations(activation, monkeypatch):
    """The autograd function around stand-ins for the kernels, with a loss whose gradient is not linear in the gate."""
    from torchturbo_b200.ops.providers import b200, native

    silu = activation == "silu"

    def kernel(x, gate, w, eps, is_silu):
        with torch.no_grad():
            return native.TorchGatedRMSNorm()(x, gate, w, eps, activation=activation), torch.ones(x.shape[0])

    def kernel_bwd(dy, x, gate, w, rstd, is_silu):
        with torch.enable_grad():
            leaves = [t.detach().requires_grad_(True) for t in (x, gate, w)]
            y = native.TorchGatedRMSNorm()(*leaves, 1e-6, activation=activation)
        return torch.autograd.grad(y, leaves, dy.detach())

    monkeypatch.setattr(b200.K, "gated_rmsnorm_fwd", kernel)
    monkeypatch.setattr(b200.K, "gated_rmsnorm_bwd", kernel_bwd)
    torch.manual_seed(0)
    start = [torch.randn(6, 64), torch.randn(6, 64), torch.rand(64)]
    probe = torch.randn(6, 64)
    res = []
    for fn in (lambda *t: b200.GatedRMSNormFn.apply(*t, 1e-6, silu), lambda *t: native.TorchGatedRMSNorm()(*t, 1e-6, activation=activation)):
        x, gate, w = (t.clone().requires_grad_(True) for t in start)
        (g,) = torch.autograd.grad(fn(x, gate, w).square().sum(), gate, create_graph=True)
        res.append([g.detach(), *torch.autograd.grad((g * probe).sum(), (x, gate, w))])
    for a, b in zip(*res):
        assert torch.allclose(a, b, atol=1e-5, rtol=1e-5)


@pytest.mark.gpu
@pytest.mark.parametrize("rows, width, activation, strided", [
    (1, 128, "silu", False), (15, 128, "sigmoid", True), (33, 64, "silu", False), (9, 256, "sigmoid", False),
    (4097, 128, "silu", True), (40000, 64, "silu", False)])
def test_gated_norm_kernel_matches_the_separate_operations(rows, width, activation, strided):
    """Same roundings as the norm kernel followed by an fp32 product, so values agree up to the last bf16 bit (2^-8 of the
    value); dw is an fp32 sum over the rows rounded once, and both sides round it: 2^-7 of its norm."""
    torch.manual_seed(rows)
    wide = torch.randn(rows, 2 * width, device="cuda").to(torch.bfloat16)
    x0, g0 = (wide[:, :width], wide[:, width:]) if strided else (wide[:, :width].contiguous(), wide[:, width:].contiguous())
    w0 = (1 + 0.1 * torch.randn(width, device="cuda")).to(torch.bfloat16)
    dy = torch.randn(rows, width, device="cuda").to(torch.bfloat16)
    outs = []
    for impl in ("b200_gated_rms_norm", "torch_gated_rms_norm"):
        x, g, w = (t.detach().requires_grad_(True) for t in (x0, g0, w0))
        y = ops.gated_rms_norm(x, g, w, 1e-6, activation=activation, impl=impl)
        y.backward(dy)
        outs.append([y, x.grad, g.grad, w.grad])
    for a, b in zip(*outs):
        a, b = a.float(), b.float()
        assert (a - b).norm() <= 2 ** -7 * b.norm(), ((a - b).norm() / b.norm())
        assert (a - b).abs().max() <= 2 ** -6 * b.abs().max()


@pytest.mark.gpu
@pytest.mark.parametrize("activation", ["silu", "sigmoid"])
@pytest.mark.parametrize("lo, hi", [(-80, -60), (-60, -30), (-30, 10)])
def test_gate_is_the_fp32_activation(activation, lo, hi):
    """Rows of +-1 normalise exactly, so values and gate gradients are those of the separate operations bit by bit unless the
    activation differs: approximate exponentials turn one bf16 value in a thousand at gates of -40."""
    gen = torch.Generator("cuda").manual_seed(0)
    rows, width = 8192, 128
    x = torch.where(torch.rand(rows, width, generator=gen, device="cuda") < 0.5, -1.0, 1.0).to(torch.bfloat16)
    gate = (torch.rand(rows, width, generator=gen, device="cuda") * (hi - lo) + lo).to(torch.bfloat16)
    w = (1 + 0.1 * torch.randn(width, generator=gen, device="cuda")).to(torch.bfloat16)
    res = []
    for impl in ("b200_gated_rms_norm", "torch_gated_rms_norm"):
        g = gate.clone().requires_grad_(True)
        y = ops.gated_rms_norm(x, g, w, 1e-6, activation=activation, impl=impl)
        y.backward(torch.full_like(y, 0.37))
        res.append((y.detach(), g.grad))
    (y, dg), (want_y, want_dg) = res
    assert torch.equal(y, want_y)
    assert (dg != want_dg).float().mean().item() <= 2 ** -20


@pytest.mark.gpu
@pytest.mark.parametrize("rows, width", [(1, 8), (31, 40), (300, 2048), (297, 1000), (5, 8192)])
def test_norm_weight_gradients_sum_every_row_once(rows, width):
    """Exact oracle: with dy = 1 and x of one value per row the weight gradient is the sum of the row signs."""
    from torchturbo_b200 import kernels as K

    x = torch.ones(rows, width, device="cuda").to(torch.bfloat16)
    x[::3] = -1
    w = torch.ones(width, device="cuda", dtype=torch.bfloat16)
    _, rstd, xs = K.rmsnorm_fwd(x, w, 0.0)
    for dtype in (torch.float32, torch.bfloat16):
        _, dw = K.rmsnorm_bwd(torch.ones_like(x), xs, w, rstd, dw_dtype=dtype)
        want = x[:, 0].float().sum()
        assert dw.dtype == dtype and dw.shape == (width,)
        assert torch.equal(dw, want.to(dtype).expand(width)), (dw, want)
