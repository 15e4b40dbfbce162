"""Operators with several outputs, when the loss reaches only some of them: against the torch formulation."""
import pytest
import torch

from torchturbo_b200.ops import ops


@pytest.mark.gpu
@pytest.mark.parametrize("use", ["first", "second", "both"])
def test_residual_norm(use):
    torch.manual_seed(0)
    leaves = [torch.randn(9, 64, device="cuda").to(torch.bfloat16), torch.randn(9, 64, device="cuda").to(torch.bfloat16),
              torch.rand(64, device="cuda").to(torch.bfloat16)]
    res = []
    for impl in ("b200_rms_norm", "torch_rms_norm"):
        x, r, w = (t.detach().requires_grad_(True) for t in leaves)
        outs = ops.rms_norm(x, w, 1e-6, residual=r, impl=impl)
        picked = dict(first=outs[:1], second=outs[1:], both=outs)[use]
        sum(t.float().sin().sum() for t in picked).backward()
        res.append([t.grad if t.grad is not None else torch.zeros_like(t) for t in (x, r, w)])
    for a, b in zip(*res):
        assert (a.float() - b.float()).norm() <= 2 ** -6 * b.float().norm() + 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("use", ["prob", "score_sum", "lse", "all"])
def test_router(use):
    torch.manual_seed(0)
    lg = torch.randn(40, 16, device="cuda")
    res = []
    for impl in ("b200_router_topk", "torch_router_topk"):
        x = lg.detach().requires_grad_(True)
        idx, prob, st = ops.router_topk(x, 3, "softmax_post", impl=impl)
        parts = dict(prob=[prob], score_sum=[st["score_sum"]], lse=[st["lse"]], all=[prob, st["score_sum"], st["lse"]])[use]
        sum(t.sin().sum() for t in parts).backward()
        res.append(x.grad)
    assert torch.allclose(*res, rtol=1e-4, atol=1e-5)


@pytest.mark.gpu
@pytest.mark.parametrize("use", ["tokens", "probs", "both"])
def test_permutation(use):
    torch.manual_seed(0)
    x0, p0 = torch.randn(50, 64, device="cuda").to(torch.bfloat16), torch.rand(50, 2, device="cuda")
    idx = torch.stack([torch.randperm(8)[:2] for _ in range(50)]).cuda()
    x, p = x0.requires_grad_(True), p0.requires_grad_(True)
    perm = ops.moe_permutation(x, idx, probs=p, num_experts=8)
    rows = perm.row_indices.reshape(-1).long()
    loss = 0.0
    if use != "probs":
        loss = loss + (perm.tokens[rows].float() * 2).sum()
    if use != "tokens":
        loss = loss + (perm.probs[rows] * 3).sum()
    loss.backward()
    assert torch.equal(x.grad, torch.full_like(x, 0.0 if use == "probs" else 4.0))
    assert torch.equal(p.grad, torch.full_like(p, 0.0 if use == "tokens" else 3.0))
