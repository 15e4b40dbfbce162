"""Backward of QK norm + RoPE over whole fused rows: value columns and weight gradients included."""
import pytest
import torch

from torchturbo_b200 import kernels as K
from torchturbo_b200.ops import ops
from torchturbo_b200.ops.providers import native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("norm", [True, False])
@pytest.mark.parametrize("T,nq,nkv", [(1, 1, 1), (7, 3, 1), (33, 4, 2), (130, 5, 5), (700, 32, 4)])
def test_against_torch(T, nq, nkv, norm):
    D = 128
    g = torch.Generator("cuda").manual_seed(T + nq)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")                                      # noqa: E731
    qkv = rnd(T, (nq + 2 * nkv) * D).bfloat16()
    wq, wk = ((1 + 0.1 * rnd(D)).bfloat16() for _ in range(2)) if norm else (None, None)
    ang = rnd(T, D // 2)
    grads = [rnd(T, h, D).bfloat16() for h in (nq, nkv)] + [rnd(T, 2 * nkv, D).bfloat16()[:, nkv:]]   # the last one strided

    def run(impl, dtype):
        x = qkv.detach().to(dtype).requires_grad_(True)
        ws = [w.detach().to(dtype).requires_grad_(True) if norm else None for w in (wq, wk)]
        out = impl(x, nq, nkv, D, *ws, ang.cos(), ang.sin(), 1e-6)
        return torch.autograd.grad(out, [x] + (ws if norm else []), [t.to(dtype) for t in grads])

    got, ref = run(ops.qk_norm_rope, torch.bfloat16), run(N.TorchQKNormRope(), torch.float32)
    assert torch.equal(got[0][:, (nq + nkv) * D:], grads[2].reshape(T, -1))
    for a, b in zip(got, ref):
        # fp32 inside the kernel and one rounding to bf16 (2^-8 relative); the torch formulation in fp32 differs by sums in another
        # order, and elements that nearly cancel are held to the size of their neighbours
        assert bool(((a.float() - b).abs() <= 2.0 ** -8 * b.abs() + 2.0 ** -9 * b.abs().mean()).all())


@pytest.mark.parametrize("norm", [True, False])
def test_value_gradients_can_be_differentiated_again(norm):
    """The value columns are passed through, so a gradient with respect to them has a gradient of its own."""
    T, nq, nkv, D = 9, 2, 1, 128
    x = torch.randn(T, (nq + 2 * nkv) * D, device="cuda").bfloat16().requires_grad_(True)
    w = torch.ones(D, device="cuda", dtype=torch.bfloat16) if norm else None
    ang = torch.randn(T, D // 2, device="cuda")
    _, _, v = ops.qk_norm_rope(x, nq, nkv, D, w, w, ang.cos(), ang.sin(), 1e-6)
    first, = torch.autograd.grad(v.float().pow(3).sum(), x, create_graph=True)
    second, = torch.autograd.grad(first.float().sum(), x)
    vx = x.detach().float()[:, (nq + nkv) * D:]
    assert bool((first[:, : (nq + nkv) * D] == 0).all()) and bool((second[:, : (nq + nkv) * D] == 0).all())
    # 3 v^2 and 6 v, rounded to bf16 once
    assert bool(((first[:, (nq + nkv) * D:].float() - 3 * vx * vx).abs() <= 2.0 ** -8 * 3 * vx * vx).all())
    assert bool(((second[:, (nq + nkv) * D:].float() - 6 * vx).abs() <= 2.0 ** -8 * 6 * vx.abs()).all())


def test_weight_gradients_in_fp32_repeat_bit_for_bit():
    T, nq, nkv, D = 500, 8, 2, 128
    qkv = torch.randn(T, 12 * D, device="cuda").bfloat16()
    w = torch.ones(D, device="cuda", dtype=torch.bfloat16)
    ang = torch.randn(T, D // 2, device="cuda")
    q, k, rstd = K.qknorm_rope_fwd(qkv, nq, nkv, D, w, w, ang.cos(), ang.sin(), 1e-6)
    runs = [K.qknorm_rope_bwd(q, k, qkv, nq, nkv, D, w, w, ang.cos(), ang.sin(), rstd, torch.zeros_like(qkv)) for _ in range(2)]
    assert runs[0][0].dtype == torch.float32 and all(torch.equal(a, b) for a, b in zip(*runs))
