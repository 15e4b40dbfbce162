"""The gated delta rule gives the same bits from version to version: the order of every fp32 sum is part of what it computes (a row's
sum over its channels in four quarters of 32, <dS, S> in the order of the rows), and its kernels use no atomics."""
import zlib

import pytest
import torch

from torchturbo_b200.ops import ops

NAMES = ("o", "state", "dq", "dk", "dv", "dg", "dbeta")
# (tokens, heads, normalised q and k, boundaries): one full chunk; ragged chunks; several documents
CASES = [(64, 1, True, None), (100, 2, False, None), (333, 4, True, [0, 120, 250, 333])]
# CRC-32 of the results' bytes
BITS = {
    (64, 1): (1225968711, 1965896267, 2395629162, 3078842440, 2998172345, 2648968121, 2499274654),
    (100, 2): (2384760309, 2226368713, 2716779617, 2568819240, 3014159632, 2218420553, 227062732),
    (333, 4): (924645152, 3718101397, 3367393727, 3574440720, 2167960796, 3851840133, 446313287),
}


def _pattern(shape, step, period, dtype=torch.bfloat16):
    """Values in [-1, 1] by whole-number arithmetic, the same with every version of every generator."""
    n = torch.Size(shape).numel()
    i = torch.arange(n, dtype=torch.int64)
    return (((i * step + i // 131 * 17) % period - period // 2).double() / (period // 2)).to(dtype).view(shape).cuda()


def checksums(T, H, l2, cu):
    size = 1.0 if l2 else 0.125
    q, k, v, do = (_pattern((1, T, H, 128), a, m) for a, m in ((7919, 2039), (104729, 1999), (15485863, 2027), (32452843, 1987)))
    q, k = q * size, k * size                                   # (a power of two: exact)
    g = -(_pattern((1, T, H), 613, 997, torch.float32) + 1) * 0.25
    beta = (_pattern((1, T, H), 331, 991, torch.float32) + 1) * 0.5
    leaves = [t.detach().requires_grad_(True) for t in (q, k, v, g, beta)]
    o, state = ops.gated_delta_rule(*leaves, use_qk_l2norm_in_kernel=l2, cu_seqlens=cu, output_final_state=True)
    grads = torch.autograd.grad((o, state), leaves, (do, torch.full_like(state, 0.0078125)))
    results = [t.detach().contiguous() for t in (o, state, *grads)]
    assert all(bool(torch.isfinite(t.float()).all()) for t in results)
    return [zlib.crc32(t.cpu().view(torch.uint8).numpy().tobytes()) for t in results]


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}x{c[1]}")
def test_bits(case):
    got = checksums(*case)
    assert dict(zip(NAMES, got)) == dict(zip(NAMES, BITS[case[:2]]))
