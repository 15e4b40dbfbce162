"""Forward attention with two query tiles per thread block, and the choice between one and two."""
import math

import pytest
import torch

from torchturbo_b200 import kernels as K


@pytest.mark.parametrize("lens,heads,width,causal,rows", [
    ([16001], 40, 128, True, 256), ([1100, 900, 1300, 796], 32, 128, True, 256), ([784, 816], 16, 72, False, 256),
    ([2048], 16, 128, True, 128), ([8192], 4, 128, True, 128), ([100, 100, 100], 8, 128, True, 128), ([784], 16, 72, False, 128),
    ([0, 5, 0], 1, 128, True, 128), ([], 1, 128, True, 128),
    ([784] * 5, 8, 128, False, 128), ([300] * 8, 8, 128, True, 256),        # the last wave decides
    ([16384], 4, 128, True, 256), ([16384], 4, 192, True, 128), ([4096], 32, 192, True, 256),
])
def test_query_rows_per_block(lens, heads, width, causal, rows):
    """Many blocks take two tiles each; where the longest blocks would decide, or the last wave, each takes one."""
    assert K.attn_tile_rows(lens, heads, causal, 148, width) == rows


def test_benchmark_takes_the_table_of_the_operator(monkeypatch):
    from torchturbo_b200.benchmarks import attention_bench

    monkeypatch.setattr(K, "num_sms", lambda *_: 148)
    monkeypatch.setattr(torch.Tensor, "cuda", lambda self: self)
    cu = torch.tensor([0, 1000, 4000, 8192], dtype=torch.int32)
    for heads, width, rows in ((32, 128, 256), (1, 128, 128), (1, 192, 128)):
        table = attention_bench._forward_table(cu, [1000, 3000, 4192], heads, width)
        assert table["tile_rows"] == rows and torch.equal(table["q_tiles_dev"], K.build_q_tiles(cu, rows)) and table["rows"] == (0, 8192)


def test_pair_table_covers_the_same_rows():
    cu = torch.tensor([3, 3, 4, 260, 516, 773, 1000], dtype=torch.int32)
    one, two = (K.build_q_tiles(cu, b).tolist() for b in (128, 256))
    covered = sorted((q, s, e) for q0, s, e in two for q in (q0, q0 + 128) if q < e)
    assert covered == sorted(map(tuple, one))


def _reference(q, k, v, cu, causal, scale):
    """fp32 result, sum of |p v| and logsumexp."""
    rep = q.shape[1] // k.shape[1]
    out, mag = torch.zeros(2, q.shape[0], q.shape[1], 128, device=q.device)
    lse = torch.full((q.shape[1], q.shape[0]), -math.inf, device=q.device)
    for a, b in zip(cu[:-1], cu[1:]):
        qq = q[a:b].float().transpose(0, 1)
        kk, vv = (t[a:b].float().repeat_interleave(rep, 1).transpose(0, 1) for t in (k, v))
        s = qq @ kk.transpose(1, 2) * scale
        if causal:
            s = s.masked_fill(torch.ones(b - a, b - a, dtype=torch.bool, device=q.device).triu(1), -math.inf)
        p = s.softmax(-1)
        out[a:b], mag[a:b] = (p @ vv).transpose(0, 1), (p @ vv.abs()).transpose(0, 1)
        lse[:, a:b] = s.logsumexp(-1)
    return out, mag, lse


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [128, 256])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("D,Hq,Hk", [(128, 4, 2), (192, 2, 2)])
@pytest.mark.parametrize("rising", [False, True])
def test_both_tile_counts(rows, causal, D, Hq, Hk, rising):
    """Documents around the tile edges.  `rising`: the keys grow along a document, so that later blocks raise a row's maximum
    and the accumulator is rescaled."""
    lens = [1, 127, 128, 129, 255, 256, 257, 384, 385, 640, 900]
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    T = cu[-1] + 5                                      # rows behind the last boundary read as zero
    g = torch.Generator("cuda").manual_seed(D + rows)
    q, k, v = (torch.randn(T, h, d, generator=g, device="cuda") for h, d in ((Hq, D), (Hk, D), (Hk, 128)))
    if rising:
        pos = torch.cat([torch.arange(n) for n in lens + [5]]).cuda().float()
        k = k + q[:, :Hk].sign() * (pos / 20)[:, None, None]
        q = q.abs() * 0.5 + q.sign() * 0.1
    q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    bounds = torch.tensor(cu, dtype=torch.int32)
    scale = D ** -0.5
    out, lse, ml = K.attn_fwd(q, k, v, K.build_q_tiles(bounds, rows).cuda(), scale=scale, causal=causal, want_max_logit=True,
                              rows=(cu[0], cu[-1]), tile_rows=rows)
    torch.cuda.synchronize()
    assert K.attn_status()[0] == 0
    ref, mag, ref_lse = _reference(q, k, v, cu, causal, scale)
    assert torch.equal(out[cu[-1]:], torch.zeros_like(out[cu[-1]:]))
    # probabilities are rounded to bf16 and so is the result: 8 significant bits, half a unit in the last place is 2^-8 relative;
    # scores up to about 2^7 in fp32, sums of up to 900 terms and the fp32 reference itself account for another 1e-4 of the
    # magnitudes
    bound = 2.0 ** -8 * (mag + ref.abs()) + 1e-4 * mag + 1e-6
    assert ((out.float() - ref).abs() <= bound)[: cu[-1]].all()
    assert (lse[:, : cu[-1]] - ref_lse[:, : cu[-1]]).abs().max() < 1e-4 * max(1.0, float(ref_lse[:, : cu[-1]].abs().max()))
    top = torch.stack([(q[a:b].float().transpose(0, 1) @ k[a:b].float().repeat_interleave(Hq // Hk, 1).permute(1, 2, 0) * scale)
                       .masked_fill(torch.ones(b - a, b - a, dtype=torch.bool, device="cuda").triu(1) & causal, -math.inf).amax((1, 2))
                       for a, b in zip(cu[:-1], cu[1:])]).amax(0)
    assert ml.shape == (Hq,) and bool(((ml - top).abs() <= 1e-4 * top.abs().clamp(min=1.0)).all())


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [128, 256])
@pytest.mark.parametrize("D", [128, 192])
def test_maximum_in_any_tile(rows, D):
    """The per-head maximum logit, placed in the first tile of a pair, in the second, and in a document's last rows."""
    T, H, scale = 700, 6, D ** -0.5
    g = torch.Generator("cuda").manual_seed(D)
    q, k, v = (torch.randn(T, H, d, generator=g, device="cuda").bfloat16() for d in (D, D, 128))
    for h, t in enumerate((0, 127, 128, 255, 384, 699)):
        q[t, h] = k[t, h] * 4
    cu = torch.tensor([0, T], dtype=torch.int32)
    _, _, ml = K.attn_fwd(q, k, v, K.build_q_tiles(cu, rows).cuda(), scale=scale, causal=True, want_max_logit=True, rows=(0, T), tile_rows=rows)
    top = (q.float().transpose(0, 1) @ k.float().permute(1, 2, 0) * scale).masked_fill(
        torch.ones(T, T, dtype=torch.bool, device="cuda").triu(1), -math.inf).amax((1, 2))
    assert bool(((ml - top).abs() <= 1e-4 * top.abs()).all())


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [128, 256])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("D", [72, 128, 192])
def test_longer_documents(rows, causal, D):
    """More blocks than stages many times over, and a last entry of one tile or of two, the second of them cut."""
    lens, H, Dv = [2048 + 3, 1664, 2304 + 200], 2, min(D, 128)
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    g = torch.Generator("cuda").manual_seed(D + rows)
    q, k, v = (torch.randn(cu[-1], H, d, generator=g, device="cuda").bfloat16() for d in (D, D, Dv))
    scale = D ** -0.5
    out, lse, _ = K.attn_fwd(q, k, v, K.build_q_tiles(torch.tensor(cu, dtype=torch.int32), rows).cuda(), scale=scale, causal=causal,
                             rows=(0, cu[-1]), tile_rows=rows)
    torch.cuda.synchronize()
    assert K.attn_status()[0] == 0
    ref, mag, ref_lse = _reference(q, k, torch.nn.functional.pad(v, (0, 128 - Dv)), cu, causal, scale)
    ref, mag = ref[..., :Dv], mag[..., :Dv]
    assert bool(((out.float() - ref).abs() <= 2.0 ** -8 * (mag + ref.abs()) + 1e-4 * mag + 1e-6).all())     # as above
    assert (lse - ref_lse).abs().max() < 1e-4 * float(ref_lse.abs().max())


@pytest.mark.gpu
@pytest.mark.parametrize("D", [128, 192])
@pytest.mark.parametrize("where", ["q", "k", "v"])
@pytest.mark.parametrize("value", [math.inf, -math.inf, math.nan])
def test_values_that_are_not_finite(D, where, value):
    """One element that is not finite spoils the rows that see it, and no other, with one query tile per block and with two."""
    T, H, scale, at = 900, 2, D ** -0.5, 300
    g = torch.Generator("cuda").manual_seed(D)
    args = {n: torch.randn(T, H, d, generator=g, device="cuda").bfloat16() for n, d in (("q", D), ("k", D), ("v", 128))}
    clean = {n: t.clone() for n, t in args.items()}
    args[where][at, 1, 5] = value
    cu = torch.tensor([0, 256, T], dtype=torch.int32)
    got = {}
    for rows in (128, 256):
        table = K.build_q_tiles(cu, rows).cuda()
        got[rows], ok = (K.attn_fwd(*(t[n] for n in "qkv"), table, scale=scale, causal=True, rows=(0, T), tile_rows=rows)[0].float()
                         for t in (args, clean))
        torch.cuda.synchronize()
        assert K.attn_status()[0] == 0
        touched = torch.zeros(T, H, dtype=torch.bool, device="cuda")
        touched[at: at + 1 if where == "q" else T, 1] = True
        if where == "v":      # the row block of the key at hand multiplies it by zero as well: 0 x inf is not a number
            touched[256:, 1] = True
        assert torch.equal(got[rows][~touched], ok[~touched])
    assert bool(((got[128] == got[256]) | (got[128].isnan() & got[256].isnan())).all())
    assert not bool(got[256][at:, 1].isfinite().all())
