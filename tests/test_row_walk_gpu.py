"""Backward kernels whose blocks walk rows, at row counts around the number of blocks (one row, one or two a block, a remainder) and at the
widths where threads own no column, a block has one or more warps, or runs alone on its SM, against 64 bits."""
import pytest
import torch

ROWS, WIDTHS = [1, 5, 297, 600, 1185], [8, 264, 2048, 2056, 4104, 8192]


def _near(got, want, mag, terms):
    """bf16 results of fp32 sums: half a unit of 2^-8, and 2^-24 of the summed magnitudes for each of `terms` roundings."""
    assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + mag * terms * 2.0 ** -24 + 1e-6).all()


@pytest.mark.gpu
@pytest.mark.parametrize("T", ROWS)
@pytest.mark.parametrize("H", WIDTHS)
def test_norms(T, H):
    from torchturbo_b200 import kernels as K

    g = torch.Generator("cuda").manual_seed(T * H)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()      # noqa: E731
    x, dy, res, w, b = rnd(T, H), rnd(T, H), rnd(T, H), rnd(H), rnd(H)
    X, DY, W = x.double(), dy.double(), w.double()
    _, rstd, _ = K.rmsnorm_fwd(x, w, 1e-6)
    dx, dw = K.rmsnorm_bwd(dy, x, w, rstd, dres=res, dw_dtype=torch.bfloat16)
    r = rstd.double()[:, None]
    xh, gw = X * r, DY * W
    dot = (gw * xh).mean(1, keepdim=True)
    size = r * (gw.abs() + xh.abs() * (gw * xh).abs().mean(1, keepdim=True))
    _near(dx, r * (gw - xh * dot) + res.double(), size + res.double().abs(), 64)
    _near(dw, (DY * xh).sum(0), (DY * xh).abs().sum(0), 64)
    _, mean, rstd = K.layernorm_fwd(x, w, b, 1e-6)
    dx, dw, db = K.layernorm_bwd(dy, x, w, mean, rstd, dw_dtype=torch.bfloat16)
    r = rstd.double()[:, None]
    xh = (X - mean.double()[:, None]) * r
    dot = (gw * xh).mean(1, keepdim=True)
    size = r * (gw.abs() + gw.abs().mean(1, keepdim=True) + xh.abs() * (gw * xh).abs().mean(1, keepdim=True))
    _near(dx, r * (gw - gw.mean(1, keepdim=True) - xh * dot), size, 64)
    _near(dw, (DY * xh).sum(0), (DY * xh).abs().sum(0), 64)
    _near(db, DY.sum(0), DY.abs().sum(0), 64)


@pytest.mark.gpu
@pytest.mark.parametrize("T", ROWS)
@pytest.mark.parametrize("C", [8, 4304, 8192, 8200, 16384])
def test_bias_and_activation(T, C):
    from torchturbo_b200 import kernels as K

    g = torch.Generator("cuda").manual_seed(T * C)
    x, dy, b = (torch.randn(*s, device="cuda", generator=g).bfloat16() for s in ((T, C), (T, C), (C,)))
    dx, db = K.bias_act_bwd(dy, x, b, None, db_dtype=torch.bfloat16)
    assert dx is dy
    _near(db, dy.double().sum(0), dy.double().abs().sum(0), 64)
    dx, db = K.bias_act_bwd(dy, x, b, "gelu", db_dtype=torch.bfloat16)
    z = (x.double() + b.double()).requires_grad_()
    want, = torch.autograd.grad(torch.nn.functional.gelu(z), z, dy.double())
    # the kernel's error function and exponential are good to 2^-18 of their argument's scale (|z| < 12)
    assert ((dx.double() - want).abs() <= 2.0 ** -8 * want.abs() + dy.double().abs() * 2.0 ** -14).all()
    assert ((db.double() - want.sum(0)).abs() <= 2.0 ** -8 * want.sum(0).abs() + dy.double().abs().sum(0) * 2.0 ** -14).all()


@pytest.mark.gpu
@pytest.mark.parametrize("T", [2, 148, 149, 296, 301, 591])
@pytest.mark.parametrize("H", [264, 2048, 4104, 8192])
def test_norms_with_a_row_or_two_for_a_block(T, H):
    test_norms(T, H)


@pytest.mark.gpu
@pytest.mark.parametrize("T", [2, 296])
@pytest.mark.parametrize("C", [4304, 16384])
def test_bias_and_activation_with_a_row_for_a_block(T, C):
    test_bias_and_activation(T, C)
