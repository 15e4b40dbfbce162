"""Buffers whose address goes to a C entry point outlive the call."""
import weakref

import torch

from torchturbo_b200 import kernels as K


def test_scratch_of_the_per_channel_delta_backward_is_held_during_the_call(monkeypatch):
    made, seen, empty = [], [], torch.empty

    def recording(*size, **kw):
        t = empty(*size, **kw)
        made.append((t.data_ptr(), weakref.ref(t)))
        return t

    class Lib:
        def ttb_delta_vec_bwd_post(self, *args):
            addresses = {a.value for a in args if hasattr(a, "value")}
            seen.append([ref() is not None for at, ref in made if at in addresses])
            return 0

    monkeypatch.setattr(torch, "empty", recording)
    monkeypatch.setattr(K, "lib", lambda: Lib())
    monkeypatch.setattr(K, "_stream", lambda: None)
    monkeypatch.setattr(K, "check_device", lambda t: None)
    R, H = 3, 2
    q, do = (torch.zeros(R, H, 128, dtype=torch.bfloat16) for _ in range(2))
    g, beta = torch.zeros(R, H, 128), torch.zeros(R, H)
    x, tri, st = torch.zeros(H, 1, 64, 128), torch.zeros(H, 1, 64, 64), torch.zeros(H, 2, 128, 128)
    K.delta_bwd_post(q, q, q, g, beta, torch.zeros(1, 3, dtype=torch.int32), do, tri, x, x, st, st, l2=True, scale=1.0)
    assert seen == [[True] * 4]                                  # dq, dk, dv and the scratch
