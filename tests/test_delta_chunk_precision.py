"""Precision of the fused delta-rule kernels, kernel by kernel against the same formulas in 64 bits.

Every kernel is given the fp32 tensors it reads, so what is compared is its own arithmetic.  fp32 results are held against
the error that fp32 torch products make on the same inputs.  Results that leave in bf16 are made to cancel, so that what is
left is the error of the operands and sums and not the last rounding.  An fp32 operand that entered the tensor cores as two
bf16 terms would leave 2^-17 of every product, one of three terms leaves less than an fp32 rounding."""
import pytest
import torch

D, C = 128, 64


def _case(T, H, vec, l2, seed=0, device="cuda"):
    gen = torch.Generator().manual_seed(seed * 1000 + T)
    q, k, v, do = (torch.randn(T, H, D, generator=gen).to(torch.bfloat16) for _ in range(4))
    if not l2:
        q, k = q * 0.0625, k * 0.0625
    g = -torch.rand(T, H, *([D] if vec else []), generator=gen) * 0.3
    beta = torch.rand(T, H, generator=gen)
    rows = torch.tensor([[r, min(C, T - r), 0] for r in range(0, T, C)], dtype=torch.int32)
    return [t.to(device) for t in (q, k, v, do, g, beta, rows)]


def chunk_terms(q, k, g, beta, rows, l2, scale, dtype):
    """q^, k^, beta, G and the score matrices L, A of every chunk: [H, NC, 64, ..]."""
    NC = rows.shape[0]

    def chunks(t):
        out = t.new_zeros(NC, C, *t.shape[1:])
        for c, (r, n, _) in enumerate(rows.tolist()):
            out[c, :n] = t[r:r + n]
        return out.movedim(2, 0)

    qh, kh, bc, G = chunks(q.to(dtype)), chunks(k.to(dtype)), chunks(beta.to(dtype)), chunks(g.to(dtype)).cumsum(2)
    if l2:
        qh, kh = (t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6) for t in (qh, kh))
    qh = qh * scale
    low = torch.ones(C, C, dtype=torch.bool, device=q.device).tril()
    if G.dim() == 4:
        pieces = []
        for h in range(G.shape[0]):
            Dm = (G[h, :, :, None] - G[h, :, None]).masked_fill(~low[..., None], -float("inf")).exp()
            pieces.append(torch.stack([torch.einsum("nik,nijk,njk->nij", t, Dm, kh[h]) for t in (kh[h] * bc[h, ..., None], qh[h])]))
        L, A = torch.stack(pieces, 1)
        eG, out, last = G.exp(), (G[:, :, -1:] - G).exp(), G[:, :, -1].exp()[..., None]
    else:
        Dm = (G[..., None] - G[..., None, :]).masked_fill(~low, -float("inf")).exp()
        L, A = (t @ kh.transpose(-1, -2) * Dm for t in (kh * bc[..., None], qh))
        eG, out, last = G.exp()[..., None], (G[..., -1:] - G).exp()[..., None], G[..., -1].exp()[..., None, None]
    return qh, kh, bc[..., None], eG, out, last, L.tril(-1), A, chunks


def surrogate(q, k, v, g, beta, rows, do, T, x, dx, S, dS, l2, scale, dtype):
    """Gradients of one chunk given its new values x, their gradient dx, the state S at its start and the gradient dS of the
    state at its end: (dq, dk, dv, dg, dbeta) by autograd through every place where q, k, v, g and beta enter."""
    leaves = [t.detach().to(dtype).requires_grad_(True) for t in (q, k, v, g, beta)]
    qh, kh, bc, eG, out, last, L, A, chunks = chunk_terms(leaves[0], leaves[1], leaves[3], leaves[4], rows, l2, scale, dtype)
    T, x, dx, S, dS = (t.to(dtype) for t in (T, x, dx, S, dS))
    dob = chunks(do.to(dtype))
    db = T.transpose(-1, -2) @ dx
    total = (db * bc * chunks(leaves[2])).sum() - ((db @ x.transpose(-1, -2)) * L).sum() + ((dob @ x.transpose(-1, -2)) * A).sum()
    total = total + ((dob @ S.transpose(-1, -2)) * qh * eG).sum() - ((db @ S.transpose(-1, -2)) * bc * kh * eG).sum()
    total = total + ((x @ dS.transpose(-1, -2)) * kh * out).sum() + (dS * S * last).sum()
    return torch.autograd.grad(total, leaves)


def rel(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


def stages(T, H, vec, l2, seed=0):
    """(name, kernel result, 64-bit result, fp32 torch result) of every kernel output, each from the same fp32 inputs."""
    from torchturbo_b200 import kernels as K

    q, k, v, do, g, beta, rows = _case(T, H, vec, l2, seed)
    scale, kw = D ** -0.5, dict(l2=l2, scale=D ** -0.5)
    NC = rows.shape[0]
    Tm, A, u, w, ko, decay = K.delta_prep(q, k, v, g, beta, rows, **kw)
    res = []
    forms = {}
    for dt in (torch.float64, torch.float32):
        qh, kh, bc, eG, out, last, L, A_, chunks = chunk_terms(q, k, g, beta, rows, l2, scale, dt)
        eye = torch.eye(C, dtype=dt, device=q.device).expand_as(L)
        T_ = torch.linalg.solve_triangular(eye + L, eye, upper=False, unitriangular=True)
        forms[dt] = dict(T=T_, A=A_, u=T_ @ (bc * chunks(v.to(dt))), w=T_ @ (bc * kh * eG), k_out=kh * out,
                         decay=last.reshape(decay.shape))
    got = dict(T=Tm, A=A, u=u, w=w, k_out=ko, decay=decay)
    res += [(n, got[n], forms[torch.float64][n], forms[torch.float32][n]) for n in got]
    gen = torch.Generator(q.device).manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=q.device)                                     # noqa: E731
    x, dx, S, dS = rnd(H, NC, C, D), rnd(H, NC, C, D), rnd(H, NC + 1, D, D), rnd(H, NC + 1, D, D)
    for c, (_, n, _) in enumerate(rows.tolist()):            # rows past the end of a sequence are zero on both sides
        x[:, c, n:] = 0
        dx[:, c, n:] = 0
    o = K.delta_out(q, k, v, g, beta, rows, A, x, S, **kw)
    gx, gs = K.delta_bwd_pre(q, k, v, g, beta, rows, do, A, 1, **kw)
    post = K.delta_bwd_post(q, k, v, g, beta, rows, do, Tm, x, dx, S, dS, **kw)
    for dt in (torch.float64, torch.float32):
        qh, kh, bc, eG, out, last, L, A_, chunks = chunk_terms(q, k, g, beta, rows, l2, scale, dt)
        oc = (qh * eG) @ S[:, :NC].to(dt) + A.to(dt) @ x.to(dt)
        dob = chunks(do.to(dt))
        forms[dt] = dict(o=torch.cat([oc[:, c, :n] for c, (_, n, _) in enumerate(rows.tolist())], 1).transpose(0, 1),
                         gx=A.to(dt).transpose(-1, -2) @ dob, gS=(qh * eG).transpose(-1, -2) @ dob)
        forms[dt].update(zip(("dq", "dk", "dv", "dg", "dbeta"),
                             surrogate(q, k, v, g, beta, rows, do, Tm, x, dx, S[:, :NC], dS[:, 1:], l2, scale, dt)))
    got = dict(o=o, gx=gx, gS=gs[:, :NC], **dict(zip(("dq", "dk", "dv", "dg", "dbeta"), post)))
    res += [(n, got[n], forms[torch.float64][n], forms[torch.float32][n]) for n in got]
    torch.cuda.synchronize()
    assert K.status() == (0, 0)
    return res


@pytest.mark.gpu
@pytest.mark.parametrize("vec", [False, True])
@pytest.mark.parametrize("T, H, l2", [(64, 2, True), (257, 2, False), (1, 1, True), (300, 3, True)])
def test_fp32_results_are_as_close_as_fp32_products(vec, T, H, l2):
    """Twice the error of torch in fp32 (measured: 0.4 to 1.5 times; with two-term operands dg 4 to 14 and dbeta 13 to 16
    times), and a few roundings where torch happens to be exact."""
    for name, got, want, fp32 in stages(T, H, vec, l2):
        if got.dtype == torch.float32:
            err, ref = ((t.double() - want).norm().item() for t in (got, fp32))
            assert err <= 2 * ref + 2 ** -22 * want.norm().item(), (name, err, ref)
        else:
            assert rel(got, want) <= 2 ** -9, (name, rel(got, want))


@pytest.mark.gpu
@pytest.mark.parametrize("vec", [False, True])
@pytest.mark.parametrize("which", ["state", "scores"])
def test_outputs_that_cancel_keep_fp32_operands(vec, which):
    """o = (q^ e^G) S + A x with S in the null space of q^ e^G, or x along the smallest singular vector of A: what remains is
    the operands' rounding.  fp32 dot products of 64 or 128 terms leave about 2^-25 of the sum of the absolute products (in
    norm); two-term operands leave 2^-21.5."""
    from torchturbo_b200 import kernels as K

    T, H = 128, 2
    q, k, v, do, g, beta, rows = _case(T, H, vec, True)
    kw = dict(l2=True, scale=D ** -0.5)
    A = K.delta_prep(q, k, v, g, beta, rows, **kw)[1]
    qh, kh, bc, eG = chunk_terms(q, k, g, beta, rows, True, D ** -0.5, torch.float64)[:4]
    gen = torch.Generator("cuda").manual_seed(3)
    x, S = torch.zeros(H, 2, C, D, device="cuda"), torch.zeros(H, 3, D, D, device="cuda")
    if which == "state":
        null = torch.linalg.svd(qh * eG)[2][:, :, C:]                                       # [H, NC, 64, 128]
        S[:, :2] = (null.transpose(-1, -2) @ torch.randn(H, 2, C, D, generator=gen, device="cuda").double()).float()
        left, right = qh * eG, S[:, :2].double()
    else:
        least = torch.linalg.svd(A.double())[2][:, :, -1]
        x = (least[..., None] * torch.randn(H, 2, 1, D, generator=gen, device="cuda").double()).float()
        left, right = A.double(), x.double()
    o = K.delta_out(q, k, v, g, beta, rows, A, x, S, **kw)
    want = (left @ right).reshape(H, T, D).transpose(0, 1)
    size = (left.abs() @ right.abs()).reshape(H, T, D).transpose(0, 1)
    assert want.norm() <= 2 ** -16 * size.norm()                                            # they do cancel
    assert (o.double() - want).norm() <= 2 ** -23 * size.norm() + 2 ** -8 * want.norm(), ((o.double() - want).norm() / size.norm())


@pytest.mark.gpu
@pytest.mark.parametrize("vec", [False, True])
def test_keys_that_cancel_keep_fp32_operands(vec):
    """Equal unit keys and beta = 1 make T bidiagonal and w = T (beta k^ e^G) zero from the second row on; both factors are
    fp32 values.  Entries of size 1/8 times a decay: fp32 leaves a few 2^-24 of them, two-term operands 2^-18."""
    from torchturbo_b200 import kernels as K

    q, k, v, do, g, beta, rows = _case(C, 1, False, True)
    k = torch.where(torch.arange(D, device="cuda") % 2 == 0, 0.125, 0.0).to(torch.bfloat16).expand(C, 1, D).contiguous()
    g = g.unsqueeze(-1).expand(C, 1, D).contiguous() if vec else g
    w = K.delta_prep(q, k, v, g, torch.ones_like(beta), rows, l2=False, scale=1.0)[3]
    assert (w[0, 0, 0].float() - k[0, 0].float() * g[0].exp().reshape(-1)).abs().max() <= 2 ** -8 * 0.125
    assert w[0, 0, 1:].float().norm() <= 2 ** -21 * 0.125 * (63 * 64) ** 0.5, w[0, 0, 1:].float().norm() / (0.125 * (63 * 64) ** 0.5)


@pytest.mark.gpu
@pytest.mark.parametrize("vec", [False, True])
def test_decays_are_exponentials_over_their_whole_range(vec):
    """One row per head, so the chunk's decay is exp(g) of a single number, -inf (a reset) included.  expf and exp2f are good to
    2^-22; per channel g is first rounded in units of log2, half a unit of 2^-23 of it."""
    from torchturbo_b200 import kernels as K

    x = torch.cat((torch.linspace(-110, 20, 4093), torch.tensor([0.0, -1e30, -float("inf")]))).cuda()
    H = x.numel()
    q, k, v = (torch.ones(1, H, D, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    g = x.view(1, H, 1).expand(1, H, D).contiguous() if vec else x.view(1, H)
    rows = torch.tensor([[0, 1, 0]], dtype=torch.int32, device="cuda")
    got = K.delta_prep(q, k, v, g, torch.ones(1, H, device="cuda"), rows, l2=True, scale=1.0)[5].reshape(H, -1).double()
    want = x.double().exp()[:, None]
    tol = 2 ** -22 + (x.abs().double()[:, None] * 2 ** -23 if vec else 0.0)
    normal = want >= 2 ** -126
    assert (((got - want).abs() <= tol * want) | ~normal).all()
    assert (got[(~normal).expand_as(got)] <= 2 ** -126).all() and (got[-1] == 0).all() and (got[-2] == 0).all()
