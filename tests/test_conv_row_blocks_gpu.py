"""Short convolution at row counts around its steps of four rows and around a block's share of the rows, against float64."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _oracle(x, w, dy, start):
    """(y, dx, dw) and, with every factor made positive, what their errors are measured in."""
    T, D = x.shape
    W = w.shape[1]
    t = torch.arange(T)
    tap = [((t - s >= start).nonzero().flatten(), s) for s in range(W)]          # rows that see the row s behind
    pre = torch.zeros_like(x)
    for rows, s in tap:
        pre[rows] += w[:, W - 1 - s] * x[rows - s]
    sg = torch.sigmoid(pre)
    y, d, size = pre * sg, dy * sg * (1 + pre * (1 - sg)), dy.abs() * (1 + pre.abs())
    dx, adx, dw, adw = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(w), torch.zeros_like(w)
    apre = torch.zeros_like(x)
    for rows, s in tap:
        apre[rows] += (w[:, W - 1 - s] * x[rows - s]).abs()
        dx[rows - s] += w[:, W - 1 - s] * d[rows]
        adx[rows - s] += w[:, W - 1 - s].abs() * size[rows]
        dw[:, W - 1 - s] = (d[rows] * x[rows - s]).sum(0)
        adw[:, W - 1 - s] = (size[rows] * x[rows - s].abs()).sum(0)
    return y, dx, dw, apre, adx, adw


@pytest.mark.parametrize("T", [1, 3, 4, 5, 148, 149, 593, 1201])
@pytest.mark.parametrize("D, W", [(8, 4), (520, 4), (520, 3), (4104, 4)])
def test_rows(T, D, W):
    from torchturbo_b200 import kernels as K

    g = torch.Generator().manual_seed(T * W)
    x, dy = (torch.randn(T, D, generator=g).bfloat16() for _ in range(2))
    w = (torch.randn(D, W, generator=g) * 0.5).bfloat16()
    cu = sorted({0, T, *(int(c) for c in torch.randint(0, T, (3,), generator=g))})
    start, end = torch.empty(T, dtype=torch.int32), torch.empty(T, dtype=torch.int32)
    for a, b in zip(cu, cu[1:]):
        start[a:b], end[a:b] = a, b
    X, DY, Wt, S, E = (t.cuda() for t in (x, dy, w, start, end))
    y = K.causal_conv1d_fwd(X, Wt, None, S, True)
    dx, dw, _ = K.causal_conv1d_bwd(DY, X, Wt, None, S, E, True)
    want = _oracle(x.double(), w.double(), dy.double(), start.long())
    # fp32 sums and approximate exponentials: 2^-17 of the operands' sizes.  A bf16 result has 8 significant bits, so rounding to nearest
    # moves it by at most half a unit of the last one, 2^-8 of a value just above a power of two; dx has that once more from the rows'
    # gradients, which are rounded before the products.
    for got, ref, size, rounded in ((y, want[0], want[3], 0.0), (dx, want[1], want[4], 2.0 ** -8)):
        assert ((got.double().cpu() - ref).abs() <= ref.abs() * 2.0 ** -8 + size * (2.0 ** -17 + rounded * (1 + 2.0 ** -8)) + 1e-30).all()
    assert ((dw.double().cpu() - want[2]).abs() <= want[5] * 2.0 ** -17 + 1e-30).all()


@pytest.mark.parametrize("T, D", [(2, 8200), (63, 8200), (300, 8200), (1190, 512), (1776, 1032), (6000, 2056)])
def test_rows_of_a_block(T, D):
    """Blocks of one to three rows, of one or more whole steps, and (the last) of as many as fill the chip twice."""
    test_rows(T, D, 4)
