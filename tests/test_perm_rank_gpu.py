"""Stable ranks of the expert packing against a sort, over sizes around a warp, a block round and several rounds."""
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("T, k, E", [(1, 1, 1), (1, 8, 16), (31, 1, 3), (33, 2, 256), (1024, 1, 2), (1025, 1, 5), (4097, 8, 128),
                                     (32769, 1, 7), (33000, 2, 16)])
@pytest.mark.parametrize("skew", [False, True])
def test_rows_follow_expert_then_token_order(T, k, E, skew):
    from torchturbo_b200 import kernels as K

    gen = torch.Generator().manual_seed(T + E)
    idx = torch.randint(0, E, (T, k), generator=gen)
    if skew:
        idx[: T // 2] = E - 1
    pm = K.perm_index(idx.to(torch.int32).cuda(), E)
    flat = idx.reshape(-1)
    counts = torch.bincount(flat, minlength=E)
    padded = (counts + 127) // 128 * 128
    start = torch.cat((torch.zeros(1, dtype=torch.long), padded.cumsum(0)))
    order = torch.sort(flat, stable=True).indices
    want = torch.empty_like(flat)
    want[order] = torch.arange(flat.numel()) - torch.repeat_interleave(counts.cumsum(0) - counts, counts) \
        + torch.repeat_interleave(start[:-1], counts)
    assert pm["counts"].cpu().tolist() == counts.tolist()
    assert pm["seg_start"].cpu().tolist() == start.tolist()
    assert torch.equal(pm["row_of"].cpu().long(), want)
