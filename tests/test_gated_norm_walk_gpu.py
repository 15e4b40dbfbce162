"""Gated RMSNorm at row counts around a block's rows and beyond one walk of the grid: every row against float64, and some as when they
are normalised by themselves."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H", [64, 128, 256])
@pytest.mark.parametrize("extra", [-1, 0, 1, 5])
@pytest.mark.parametrize("blocks", [1, 3, 8 * 148 * 2])
def test_rows(H, extra, blocks):
    from torchturbo_b200 import kernels as K

    per = 2048 // H
    R = blocks * per + extra
    g = torch.Generator("cuda").manual_seed(R)
    x, gate, dy = (torch.randn(R, H, generator=g, device="cuda").bfloat16() for _ in range(3))
    w = torch.randn(H, generator=g, device="cuda").bfloat16()
    y, rstd = K.gated_rmsnorm_fwd(x, gate, w, 1e-6, True)
    dx, dgate, dw = K.gated_rmsnorm_bwd(dy, x, gate, w, rstd, True)
    xd, gd, dd, wd = x.double(), gate.double(), dy.double(), w.double()
    n = (xd * rstd.double()[:, None])
    # d(w) adds dn * n; dn is rounded to bf16 (8 significant bits, at most 2^-8 of a value), and so is the sum
    dn = dd * gd * torch.sigmoid(gd)
    size, want = (dn * n).abs().sum(0), (dn * n).sum(0)
    assert ((dw.double() - want).abs() <= size * 2.0 ** -8 * 1.01 + want.abs() * 2.0 ** -8).all()
    assert (rstd.double() * (xd.square().mean(1) + 1e-6).sqrt() - 1).abs().max() <= 2.0 ** -20
    # every row: x * rstd, its product with w, and the result are each rounded to bf16, u = 2^-8 of a value at most; fp32 between them
    # adds 2^-18 of the operands' sizes
    u, small = 2.0 ** -8 * 1.02, 2.0 ** -18
    r = (xd.square().mean(1, keepdim=True) + 1e-6).rsqrt()
    sg = torch.sigmoid(gd)
    act, slope, xh = gd * sg, sg * (1 + gd * (1 - sg)), xd * r
    assert ((y.double() - xh * wd * act).abs() <= (xh * wd * act).abs() * (3 * u + small)).all()
    want, size = dd * xh * wd * slope, (dd * xh * wd).abs()
    assert ((dgate.double() - want).abs() <= want.abs() * 3 * u + size * small).all()
    # dy * act is rounded before its product with w, and so is dx
    dxh = dd * act * wd
    want = r * (dxh - xh * (dxh * xh).mean(1, keepdim=True))
    size = r * (dxh.abs() + xh.abs() * (dxh * xh).abs().mean(1, keepdim=True))
    assert ((dx.double() - want).abs() <= want.abs() * u + size * (u + small)).all()
    for at in sorted({0, max(R // 2 - 1, 0), max(R - 3, 0)}):
        part = slice(at, min(at + 3, R))
        y1, r1 = K.gated_rmsnorm_fwd(x[part].clone(), gate[part].clone(), w, 1e-6, True)
        dx1, dg1, _ = K.gated_rmsnorm_bwd(dy[part].clone(), x[part].clone(), gate[part].clone(), w, r1, True)
        assert torch.equal(y[part], y1) and torch.equal(rstd[part], r1)
        assert torch.equal(dx[part], dx1) and torch.equal(dgate[part], dg1)
