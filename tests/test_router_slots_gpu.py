"""Router selection at expert counts around a warp's slots, with equal, infinite and undefined logits, against a stable sort."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E", [1, 2, 31, 32, 33, 64, 65, 127, 128, 129, 255, 256])
@pytest.mark.parametrize("k", [1, 8, 16])
def test_selection(E, k):
    from torchturbo_b200 import kernels as K

    k = min(k, E)
    g = torch.Generator().manual_seed(E * 17 + k)
    x = torch.randn(203, E, generator=g)
    x[1::4] = torch.randint(-2, 3, (x[1::4].shape[0], E), generator=g).float() * 0.5     # equal logits
    x[2, : E // 2] = float("-inf")
    x[3, 0], x[3, -1] = -0.0, 0.0
    x[5] = float("nan")
    x[6] = -torch.rand(E, generator=g) - 1
    bias = torch.randn(E, generator=g) * 0.1
    got = K.router_fwd(x.cuda(), k, "softmax_post", want_stats=True)
    order = torch.sort(torch.where(x.isnan(), float("-inf"), x), dim=1, descending=True, stable=True).indices[:, :k]
    assert torch.equal(got["topk_idx"].cpu().long(), order)
    ok = torch.arange(203) != 5
    w = torch.softmax(x.double().gather(1, order), -1)
    ok &= w.isfinite().all(1)
    # exponentials and one division in fp32
    assert ((got["topk_prob"].cpu().double() - w)[ok].abs() <= w[ok] * 2.0 ** -18 + 2.0 ** -30).all()
    assert torch.equal(got["counts"].cpu().long(), torch.bincount(order.flatten(), minlength=E))
    assert torch.equal(got["aux_counts"].cpu(), got["counts"].cpu())
    # selection by a biased score, statistics by the score itself; k distinct experts in falling order of what was sorted
    biased = K.router_fwd(x[6:].cuda().contiguous(), k, "sigmoid", expert_bias=bias.cuda(), want_stats=True)
    score = torch.sigmoid(x[6:].double())
    picked = biased["topk_idx"].cpu().long()
    assert (picked.sort(1).values.diff(dim=1) > 0).all()
    by = (score + bias.double()).gather(1, picked)
    best = (score + bias.double()).topk(k, 1).values
    assert (by - best).abs().max() <= 2.0 ** -18
    assert biased["aux_counts"].sum().item() == picked.numel()
