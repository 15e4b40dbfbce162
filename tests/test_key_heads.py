"""Gated delta rule with key heads that serve several value heads each: the same as with the key heads repeated."""
import pytest
import torch

from torchturbo_b200.ops import OpDispatcher, OpPolicy, ops
from torchturbo_b200.ops.providers.native_linear_attention import TorchGatedDeltaRule, repeat_key_heads


def _inputs(T, H, rep, device, dtype):
    g = torch.Generator(device).manual_seed(T * H * rep)
    rnd = lambda *s: torch.randn(*s, generator=g, device=device)                                      # noqa: E731
    mixed = rnd(1, T, 2 * (H // rep) * 128 + H * 128).to(dtype)
    q, k, v = mixed.split([H // rep * 128, H // rep * 128, H * 128], -1)                              # strided rows, as the mixers have them
    q, k, v = q.reshape(1, T, H // rep, 128), k.reshape(1, T, H // rep, 128), v.reshape(1, T, H, 128)
    gate = -torch.rand(1, T, H, generator=g, device=device)
    beta = torch.rand(1, T, H, generator=g, device=device)
    return [t.detach() for t in (q, k, v, gate, beta)], rnd(1, T, H, 128).to(dtype)


def _run(rule, args, do, cu, rep, repeat):
    q, k, v, g, b = (t.detach().requires_grad_(True) for t in args)
    kw = dict(use_qk_l2norm_in_kernel=True, cu_seqlens=cu, output_final_state=True)
    if repeat:
        o, fin = rule(repeat_key_heads(q, rep), repeat_key_heads(k, rep), v, g, b, **kw)
    else:
        o, fin = rule(q, k, v, g, b, heads_per_key=rep, **kw)
    return (o.detach(), fin.detach(), *torch.autograd.grad(o, (q, k, v, g, b), do))


def test_torch_formulation():
    args, do = _inputs(40, 4, 2, "cpu", torch.float32)
    cu = torch.tensor([0, 25, 40], dtype=torch.int32)
    for a, b in zip(_run(TorchGatedDeltaRule(), args, do, cu, 2, False), _run(TorchGatedDeltaRule(), args, do, cu, 2, True)):
        assert torch.equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,H,rep", [(1, 2, 2), (64, 4, 4), (130, 6, 3), (333, 4, 2)])
def test_kernels(T, H, rep, dtype):
    assert type(OpDispatcher(OpPolicy.AUTO).resolve("gated_delta_rule")).__name__ == "B200GatedDeltaRule"
    args, do = _inputs(T, H, rep, "cuda", dtype)
    cu = [0, T // 3, T] if T > 3 else [0, T]
    got, ref = (_run(ops.gated_delta_rule, args, do, cu, rep, repeat) for repeat in (False, True))
    for i, (a, b) in enumerate(zip(got, ref)):
        assert a.shape == b.shape
        if i in (2, 3) and rep > 2 or dtype == torch.float32:      # sums of three heads and more may be taken in another order
            assert float((a.float() - b.float()).abs().max()) <= 2.0 ** -7 * float(b.float().abs().max())
        else:
            assert torch.equal(a, b)
