"""Attention gradients where a key tile ends in another document, in a document's last rows or at the end of the tensor, for results that
are written once (as many key as query heads) and for sums over a group of query heads, against 64 bits."""
import pytest
import torch


def _exact(q, k, v, do, out, cu, causal, scale):
    """Gradients in 64 bits and, for each, the magnitude that its roundings are relative to: P and dS are rounded to bf16 (2^-9 of
    themselves), and Delta = rowsum(dO O) is formed from the rounded output (2^-9 of its terms)."""
    rep = q.shape[1] // k.shape[1]
    q, k, v, do, out = (t.double() for t in (q, k.repeat_interleave(rep, 1), v.repeat_interleave(rep, 1), do, out))
    grads, mags = [[torch.zeros_like(t) for t in (q, k, v)] for _ in range(2)]
    for a, b in zip(cu[:-1], cu[1:]):
        Q, K, V, dO, O = (t[a:b].transpose(0, 1) for t in (q, k, v, do, out))
        S = Q @ K.transpose(1, 2) * scale
        if causal:
            S = S.masked_fill(torch.ones(b - a, b - a, dtype=torch.bool, device=S.device).triu(1), float("-inf"))
        P, dP = S.softmax(-1), dO @ V.transpose(1, 2)
        dS = P * (dP - (P * dP).sum(-1, keepdim=True)) * scale
        mS = P * (dP.abs() + (P * dP).sum(-1, keepdim=True).abs() + (dO.abs() * O.abs()).sum(-1, keepdim=True)) * scale
        for x, val, mag in zip(range(3), (dS @ K, dS.transpose(1, 2) @ Q, P.transpose(1, 2) @ dO),
                               (mS @ K.abs(), mS.transpose(1, 2) @ Q.abs(), P.transpose(1, 2) @ dO.abs())):
            grads[x][a:b], mags[x][a:b] = val.transpose(0, 1), mag.transpose(0, 1)
    for x in (1, 2):
        T, H, D = grads[x].shape
        grads[x], mags[x] = (t.view(T, H // rep, rep, D).sum(2) for t in (grads[x], mags[x]))
    return grads, mags


@pytest.mark.gpu
@pytest.mark.parametrize("lens", [[1], [128], [65, 63], [129, 1, 126], [31, 33, 200, 97], [300]])
@pytest.mark.parametrize("Hq, Hk", [(2, 2), (6, 2)])
@pytest.mark.parametrize("D, Dv", [(128, 128), (72, 72), (64, 64), (8, 128), (192, 128)])
@pytest.mark.parametrize("causal, deterministic", [(True, False), (False, False), (True, True)])
def test_gradients(lens, Hq, Hk, D, Dv, causal, deterministic):
    from torchturbo_b200 import kernels as K
    from torchturbo_b200.ops.providers import b200_attention as BA

    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    T, gen = cu[-1], torch.Generator().manual_seed(sum(lens) + D)
    q, k, v, do = ((torch.randn(*s, generator=gen)).bfloat16().cuda() for s in ((T, Hq, D), (T, Hk, D), (T, Hk, Dv), (T, Hq, Dv)))
    tiles = BA._tiles_for(torch.tensor(cu, dtype=torch.int32), q.device)
    out, lse, _ = K.attn_fwd(q, k, v, tiles.q[128], scale=D ** -0.5, causal=causal, rows=tiles.rows)
    got = K.attn_bwd(do, q, k, v, out, lse, tiles.kv, scale=D ** -0.5, causal=causal, q_tiles_dev=tiles.q[128], rows=tiles.rows,
                     deterministic=deterministic)
    want, mags = _exact(q, k, v, do, out, cu, causal, D ** -0.5)
    for g, w, m in zip(got, want, mags):
        # two roundings of 2^-9 and the result's own, doubled for what they multiply into one another
        assert ((g.double() - w).abs() <= 2.0 ** -7 * (m + w.abs()) + 1e-6).all()
    assert K.status() == (0, 0)
