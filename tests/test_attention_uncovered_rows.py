"""Rows that no sequence covers read as zero in the output and in every gradient; covered rows do not depend on them."""
import pytest
import torch

from torchturbo_b200.ops import ops


@pytest.mark.gpu
@pytest.mark.parametrize("heads, kv_heads, D", [(4, 2, 128), (2, 2, 128), (2, 2, 192)])
@pytest.mark.parametrize("cu, T", [([0, 130, 300], 300), ([0, 130, 131], 200), ([17, 140], 260), ([5, 5, 5], 140), ([0, 0, 128, 128], 128)])
def test_uncovered_rows_are_zero(heads, kv_heads, D, cu, T):
    torch.manual_seed(T)
    junk = [torch.full((T, 8, 256), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(6)]
    del junk                                            # recycled blocks hold NaN: a row that is not written shows
    q, k, v = (torch.randn(T, h, d, device="cuda").to(torch.bfloat16).requires_grad_(True)
               for h, d in ((heads, D), (kv_heads, D), (kv_heads, 128)))
    o = ops.attention(q, k, v, torch.tensor(cu, dtype=torch.int32), causal=True)
    o.backward(torch.ones_like(o))
    covered = torch.zeros(T, dtype=torch.bool)
    for a, b in zip(cu[:-1], cu[1:]):
        covered[a:b] = True
    for t in (o, q.grad, k.grad, v.grad):
        assert torch.isfinite(t.float()).all()
        assert bool((t[~covered.cuda()] == 0).all())
