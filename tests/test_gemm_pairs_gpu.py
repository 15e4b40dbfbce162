"""Products whose 256-row tiles two thread blocks share, around the tile edges, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    from torchturbo_b200 import kernels

    assert kernels.available()
    return kernels


def _rand(*shape):
    return torch.randn(*shape, device="cuda").bfloat16()


def _sum_error(terms):
    """Unit normal factors: a sum moves by at most a unit in the last place (2^-23) of its largest value, within 5 sqrt(terms), for
    each of the terms / 16 products that the tensor cores add to it, here at least four."""
    return max(terms / 16, 4) * 2.0 ** -23 * 5 * max(terms, 16) ** 0.5


def _check(got, ref, terms):
    """`ref` in 64 bits; a bf16 result adds half a unit in its last place (2^-8 of the value, generously)."""
    bound = 2.0 ** -8 * ref.abs() + _sum_error(terms)
    diff = (got.double() - ref).abs()
    assert bool((diff <= bound).all()), float((diff - bound).max())


# Two thread blocks share a tile from 48 k-blocks of 64 per block on: one tile and its remainders; pieces along K (the last but one);
# two waves of short runs.  (384, 512, 200) stays with single blocks.
SIZES = [(136, 136, 3080), (256, 256, 3072), (264, 264, 3144), (392, 520, 3200), (384, 512, 200), (1000, 2056, 6216), (4872, 1032, 1544)]


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("M,N,Kd", SIZES)
def test_dense(K, M, N, Kd, a_mn, b_mn):
    torch.manual_seed(M + Kd)
    a, b = _rand(M, Kd), _rand(N, Kd)
    ref = a.double() @ b.double().t()
    args = (a.t().contiguous() if a_mn else a, b.t().contiguous() if b_mn else b)
    kw = dict(a_mn=a_mn, b_mn=b_mn)
    _check(K.gemm(*args, **kw), ref, Kd)
    out = torch.randn(M, N, device="cuda")
    base = out.clone()
    K.gemm(*args, out=out, accumulate=True, **kw)
    assert float((out - (base + ref)).abs().max()) <= _sum_error(Kd) + 2.0 ** -15       # and one rounding of a sum below 512
    res = _rand(M, N)
    _check(K.gemm(*args, residual=res, **kw), ref + res.double(), Kd)
    half = torch.tensor([-0.375], device="cuda")
    _check(K.gemm(*args, alpha=half, **kw), -0.375 * ref, Kd)
    out = base.clone()
    K.gemm(*args, out=out, accumulate=True, alpha=half, **kw)
    assert float((out - (base - 0.375 * ref)).abs().max()) <= _sum_error(Kd) + 2.0 ** -15
    wide = torch.full((M, N + 16), 7.0, device="cuda", dtype=torch.bfloat16)     # rows further apart: nothing beside them is written
    K.gemm(*args, out=wide[:, :N], **kw)
    _check(wide[:, :N], ref, Kd)
    assert bool((wide[:, N:] == 7).all())
    assert K.status()[0] == 0


def test_one_launch_after_another(K):
    """Products with fewer k-blocks than stages, as many and more, whose blocks end and start beside each other: the last signals of
    one may not reach the next."""
    torch.manual_seed(0)
    cases = []
    for M, N, Kd in ((256, 128 * 128, 3072), (512, 74 * 256, 64 * 48), (304, 304, 3080), (9600, 2048, 384)):
        a, b = _rand(M, Kd), _rand(N, Kd)
        cases.append((a, b, K.gemm(a, b)))
    got = [K.gemm(a, b) for _ in range(20) for a, b, _ in cases]
    torch.cuda.synchronize()
    assert K.status()[0] == 0
    for i, o in enumerate(got):
        assert torch.equal(o, cases[i % len(cases)][2])


@pytest.mark.parametrize("M,F,Kd", [(136, 64, 3080), (300, 200, 3072), (520, 328, 3144), (300, 200, 64)])
def test_swiglu(K, M, F, Kd):
    torch.manual_seed(F)
    x, w, scale = _rand(M, Kd), _rand(2 * F, Kd), torch.rand(M, device="cuda")
    pre = torch.empty(M, 2 * F, device="cuda", dtype=torch.bfloat16)
    y = K.gemm(x, w, swiglu=True, preact=pre, row_scale=scale)
    _check(pre, x.double() @ w.double().t(), Kd)
    g, u = pre.float().chunk(2, -1)
    ref = torch.nn.functional.silu(g) * u * scale[:, None]
    assert bool(((y.float() - ref).abs() <= 2.0 ** -7 * ref.abs() + 1e-6).all())       # fast exponential and division, one rounding


@pytest.mark.parametrize("counts", [[128, 0, 256, 64], [64], [0, 0], [640, 128, 0, 192, 320]])
def test_row_groups(K, counts):
    """One product per row range; an empty range gives zeros."""
    M, N = 392, 520
    torch.manual_seed(sum(counts))
    R = max(sum(counts), 64)
    a, b = _rand(R, M), _rand(R, N)
    edges = torch.tensor([0] + counts, device="cuda").cumsum(0).int()
    out = K.gemm(a, b, a_mn=True, b_mn=True, group_rows=edges)
    e = edges.tolist()
    for g in range(len(counts)):
        _check(out[g], a[e[g]:e[g + 1]].double().t() @ b[e[g]:e[g + 1]].double(), counts[g])
