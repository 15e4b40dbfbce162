"""Gradients that are contiguous but start between two 16-byte boundaries (a piece of a concatenation) are copied before a
kernel reads them sixteen bytes at a time, and the entry points refuse such addresses."""
import ctypes as C

import pytest
import torch

from torchturbo_b200 import kernels as K


def _offset(*shape):
    n = torch.Size(shape).numel()
    return torch.arange(n + 3, dtype=torch.float32).to(torch.bfloat16)[3:].view(shape)


def test_gated_norm_copies_an_offset_gradient(monkeypatch):
    from torchturbo_b200.ops.providers.b200 import GatedRMSNormFn

    seen = []

    def bwd(dy, x, gate, w, rstd, silu):
        seen.append((dy.data_ptr() % 16, dy.clone()))
        return torch.zeros_like(x), torch.zeros_like(gate), torch.zeros_like(w)

    monkeypatch.setattr(K, "gated_rmsnorm_fwd", lambda x, gate, w, eps, silu: (x * 1, torch.ones(x.shape[0])))
    monkeypatch.setattr(K, "gated_rmsnorm_bwd", bwd)
    x, gate = (torch.randn(5, 64).to(torch.bfloat16).requires_grad_(True) for _ in range(2))
    y = GatedRMSNormFn.apply(x, gate, torch.ones(64, dtype=torch.bfloat16), 1e-6, True)
    dy = _offset(5, 64)
    assert dy.is_contiguous() and dy.data_ptr() % 16
    y.backward(dy)
    assert [a for a, _ in seen] == [0] and torch.equal(seen[0][1], dy)


def test_delta_rule_copies_an_offset_gradient(monkeypatch):
    from torchturbo_b200.ops.providers.b200_linear_attention import ChunkDelta

    T, seen, z = 4, [], torch.zeros

    def pre(q, k, v, g, beta, rows, do, A, nseq, **kw):
        seen.append((do.data_ptr() % 16, do.clone()))
        return z(1, 1, 64, 128), z(1, 2, 128, 128)

    monkeypatch.setattr(K, "delta_prep", lambda *a, **kw: (z(1, 1, 64, 64), z(1, 1, 64, 64), z(1, 1, 64, 128), z(1), z(1), z(1, 1)))
    monkeypatch.setattr(K, "delta_state_scan", lambda *a, **kw: (z(1, 1, 64, 128), z(1, 2, 128, 128)))
    monkeypatch.setattr(K, "delta_out", lambda q, *a, **kw: q * 1)
    monkeypatch.setattr(K, "delta_bwd_pre", pre)
    monkeypatch.setattr(K, "delta_bwd_post", lambda q, k, v, g, beta, *a, **kw: tuple(torch.zeros_like(t) for t in (q, k, v, g, beta)))
    q, k, v = (torch.randn(T, 1, 128).to(torch.bfloat16).requires_grad_(True) for _ in range(3))
    tables = (torch.tensor([[0, 1]]), torch.tensor([[0, T, 0]]), torch.tensor([1]), torch.tensor([0]))
    o, _ = ChunkDelta.apply(q, k, v, z(T, 1), z(T, 1), None, tables, 1.0, True)
    do = _offset(T, 1, 128)
    o.backward(do)
    assert [a for a, _ in seen] == [0] and torch.equal(seen[0][1], do)


@pytest.mark.parametrize("bad", range(4))
def test_entry_points_refuse_odd_addresses(bad):
    """Refused on the host, before anything is launched, so the addresses need not exist."""
    if not K.is_built():
        pytest.skip("library not built")
    at = [C.c_void_p(4096 + (8 if i == bad else 0)) for i in range(4)]
    p = C.c_void_p(4096)
    none = C.c_void_p(0)
    assert K.lib().ttb_gated_rmsnorm_fwd(*at, p, C.c_longlong(1), 64, C.c_float(1e-6), 1, 1, none) == 902
    assert K.lib().ttb_gated_rmsnorm_bwd(*at, p, p, p, p, p, C.c_longlong(1), 64, 1, 1, none) == 902
    odd = [C.c_void_p(4096 + (4 if i == bad else 0)) for i in range(4)]
    assert K.lib().ttb_rope(odd[0], C.c_longlong(64), C.c_longlong(64), odd[1], odd[2], odd[3], C.c_longlong(1), 1, 32, C.c_float(1.0), none) == 902
