"""Ways a product leaves the GEMM kernel: plain bf16 rows through the copy engine, everything else by ordinary stores, at the edges of
a tile, into rows of a wider matrix, and for groups without rows."""
import pytest
import torch


def _rand(gen, *shape):
    return (torch.randn(*shape, generator=gen) * 0.5).bfloat16().cuda()


def _near(got, want, mag):
    """One rounding to the output type of a sum kept in fp32: half a unit of its last place, and 2^-24 of the summed magnitudes for
    every one of its (at most 2^9) partial sums."""
    unit = 2.0 ** -8 if got.dtype == torch.bfloat16 else 2.0 ** -23
    assert (got.double() - want).abs().le(want.abs() * unit + mag * 2.0 ** -15 + 1e-30).all()


@pytest.mark.gpu
@pytest.mark.parametrize("M, N", [(1, 8), (31, 64), (33, 72), (127, 128), (128, 136), (129, 200), (160, 256), (257, 264), (300, 456)])
@pytest.mark.parametrize("K", [64, 136])
def test_edges_and_wider_rows(M, N, K):
    from torchturbo_b200 import kernels as Kn

    gen = torch.Generator().manual_seed(M * N + K)
    a, b = _rand(gen, M, K), _rand(gen, N, K)
    ref, mag = a.double() @ b.double().t(), a.double().abs() @ b.double().abs().t()
    _near(Kn.gemm(a, b), ref, mag)
    for dtype in (torch.bfloat16, torch.float32):
        wide = torch.full((M + 1, N + 24), 7.0, dtype=dtype, device="cuda")
        Kn.gemm(a, b, out=wide[:M, 8:8 + N])
        _near(wide[:M, 8:8 + N], ref, mag)
        assert (wide[M] == 7).all() and (wide[:, :8] == 7).all() and (wide[:, 8 + N:] == 7).all()
        wide[:M, 8:8 + N] = 1.0
        Kn.gemm(a, b, out=wide[:M, 8:8 + N], accumulate=True)
        _near(wide[:M, 8:8 + N], ref + 1, mag + 1)
        assert (wide[M] == 7).all() and (wide[:, :8] == 7).all() and (wide[:, 8 + N:] == 7).all()
    res = _rand(gen, M, N)
    _near(Kn.gemm(a, b, residual=res), ref + res.double(), mag + res.double().abs())
    assert Kn.status() == (0, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("M, N", [(64, 8), (136, 264), (384, 512)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_groups_with_and_without_rows(M, N, dtype):
    from torchturbo_b200 import kernels as Kn

    rows = [0, 128, 0, 64, 256, 0]
    edges = torch.tensor([0] + rows).cumsum(0).to(torch.int32)
    gen = torch.Generator().manual_seed(M)
    a, b = _rand(gen, int(edges[-1]), M), _rand(gen, int(edges[-1]), N)
    out = torch.full((len(rows), M + 8, N), 7.0, dtype=dtype, device="cuda")      # groups further apart than their rows
    Kn.gemm(a, b, a_mn=True, b_mn=True, group_rows=edges.cuda(), out=out[:, :M])
    assert (out[:, M:] == 7).all()
    for g, n in enumerate(rows):
        x, y = (t[edges[g]: edges[g] + n].double() for t in (a, b))
        _near(out[g, :M], x.t() @ y, x.abs().t() @ y.abs())
    assert Kn.status() == (0, 0)
