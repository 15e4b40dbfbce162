"""The chunk recurrence of the delta rule over many short, empty and unequal sequences (more than the blocks of a launch, more than are
sorted by length), with every combination of a first state and added gradients, against 64 bits."""
import pytest
import torch


def _scan(a, b, u, dec, init, add, lens, reverse, s1, s2):
    a, b, u, dec = (t.double() for t in (a, b, u, dec))
    H, NC, ns = u.shape[0], u.shape[1], len(lens)
    if dec.dim() == 2:
        dec = dec[..., None].expand(H, NC, 128)
    X, states = torch.zeros_like(u), torch.zeros(H, NC + ns, 128, 128, dtype=torch.float64, device=u.device)
    c0 = 0
    for s, n in enumerate(lens):
        order = range(c0 + n - 1, c0 - 1, -1) if reverse else range(c0, c0 + n)
        first = (c0 + n if reverse else c0) + s
        S = add[:, first].double() if reverse else init[:, s].double() if init is not None else torch.zeros_like(states[:, 0])
        states[:, first] = S
        for c in order:
            slot = (c if reverse else c + 1) + s
            X[:, c] = u[:, c] + s1 * a[:, c] @ S
            S = dec[:, c, :, None] * S + s2 * b[:, c].transpose(1, 2) @ X[:, c] + (add[:, slot].double() if add is not None else 0)
            states[:, slot] = S
        c0 += n
    return X, states


@pytest.mark.gpu
@pytest.mark.parametrize("H, lens", [(1, [1]), (2, [3, 0, 5]), (3, [i % 4 for i in range(40)]), (5, [2] * 17), (1, [0] * 33 + [6])])
@pytest.mark.parametrize("vec", [False, True])
@pytest.mark.parametrize("with_init, with_add, reverse", [(False, False, False), (True, False, False), (False, True, False), (True, True, False),
                                                          (False, True, True)])
def test_against_64_bits(H, lens, vec, with_init, with_add, reverse):
    from torchturbo_b200 import kernels as K

    NC, ns, g = sum(lens), len(lens), torch.Generator("cuda").manual_seed(len(lens))
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)      # noqa: E731
    a, b = (rnd(H, NC, 64, 128) * 0.03).bfloat16(), (rnd(H, NC, 64, 128) * 0.03).bfloat16()
    u, dec = rnd(H, NC, 64, 128), torch.rand(*((H, NC, 128) if vec else (H, NC)), device="cuda", generator=g)
    init = rnd(H, ns, 128, 128) if with_init else None
    add = rnd(H, NC + ns, 128, 128) if with_add else None
    cu = torch.tensor([0] + lens).cumsum(0)
    seq = torch.stack((cu[:-1], torch.tensor(lens)), 1).to(torch.int32).cuda()
    s1, s2 = (1.0, -1.0) if reverse else (-1.0, 1.0)
    x, states = K.delta_state_scan(a, b, u, dec, init, add, seq, reverse=reverse, s1=s1, s2=s2)
    want_x, want_s = _scan(a, b, u, dec, init, add, lens, reverse, s1, s2)
    # S and X enter the products rounded to bf16 (2^-9 of each element), a chunk after the other, and nothing grows from chunk to chunk
    bound = 2.0 ** -8 * max(lens)
    for got, want in ((x, want_x), (states, want_s)):
        assert (got.double() - want).norm() <= bound * want.norm()
    again = K.delta_state_scan(a, b, u, dec, init, add, seq, reverse=reverse, s1=s1, s2=s2)
    assert torch.equal(x, again[0]) and torch.equal(states, again[1])


@pytest.mark.gpu
@pytest.mark.parametrize("H, lens", [(2, [3, 0, 5]), (3, [i % 4 for i in range(40)])])
def test_a_first_state_of_zero_is_not_read(H, lens):
    from torchturbo_b200 import kernels as K

    NC, ns, g = sum(lens), len(lens), torch.Generator("cuda").manual_seed(1)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)      # noqa: E731
    a, b = (rnd(H, NC, 64, 128) * 0.03).bfloat16(), (rnd(H, NC, 64, 128) * 0.03).bfloat16()
    u, dec, add = rnd(H, NC, 64, 128), torch.rand(H, NC, device="cuda", generator=g), rnd(H, NC + ns, 128, 128)
    cu = torch.tensor([0] + lens).cumsum(0)
    seq = torch.stack((cu[:-1], torch.tensor(lens)), 1).to(torch.int32).cuda()
    last = (cu[1:] + torch.arange(ns)).cuda()
    kw = dict(reverse=True, s1=1.0, s2=-1.0)
    want = K.delta_state_scan(a, b, u, dec, None, add.index_fill(1, last, 0.0), seq, **kw)
    got = K.delta_state_scan(a, b, u, dec, None, add.index_fill(1, last, float("nan")), seq, zero_first=True, **kw)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.gpu
@pytest.mark.parametrize("H, lens", [(1, [1]), (2, [1, 0, 1]), (3, [1] * 40), (5, [2] * 17), (30, [3, 3, 2, 3]), (148, [2]), (60, [2] * 4), (37, [4] * 7), (32, [4, 3, 3, 3])])
@pytest.mark.parametrize("vec", [False, True])
@pytest.mark.parametrize("with_init", [False, True])
def test_forward_with_the_longest_sequence_known(H, lens, vec, with_init):
    """Sequences of one chunk, and pairs of heads and sequences that fill the chip once or twice, take the other form of the forward pass."""
    from torchturbo_b200 import kernels as K

    NC, ns, g = sum(lens), len(lens), torch.Generator("cuda").manual_seed(H)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)      # noqa: E731
    a, b = (rnd(H, NC, 64, 128) * 0.03).bfloat16(), (rnd(H, NC, 64, 128) * 0.03).bfloat16()
    u, dec = rnd(H, NC, 64, 128), torch.rand(*((H, NC, 128) if vec else (H, NC)), device="cuda", generator=g)
    init = rnd(H, ns, 128, 128) if with_init else None
    cu = torch.tensor([0] + lens).cumsum(0)
    seq = torch.stack((cu[:-1], torch.tensor(lens)), 1).to(torch.int32).cuda()
    kw = dict(reverse=False, s1=-1.0, s2=1.0)
    x, states = K.delta_state_scan(a, b, u, dec, init, None, seq, longest=max(lens), **kw)
    want_x, want_s = _scan(a, b, u, dec, init, None, lens, False, -1.0, 1.0)
    bound = 2.0 ** -8 * max(lens)                   # as above
    for got, want in ((x, want_x), (states, want_s)):
        assert (got.double() - want).norm() <= bound * want.norm()
    other = K.delta_state_scan(a, b, u, dec, init, None, seq, **kw)
    assert torch.equal(x, other[0]) and torch.equal(states, other[1])
    assert K.status() == (0, 0)
