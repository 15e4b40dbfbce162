"""lm_head + cross entropy in one piece against the chunked accumulation, and the scaled GEMM store it relies on."""
import pytest
import torch

from torchturbo_b200.ops import ops


@pytest.mark.gpu
@pytest.mark.parametrize("T, H, V, chunk", [(1, 64, 128, 4), (130, 128, 1000, 64), (257, 128, 1000, 64), (200, 64, 520, 512), (256, 128, 1032, 100)])
@pytest.mark.parametrize("scale", [1.0, 0.37])
def test_whole_and_chunked_forms_agree_with_fp64(T, H, V, chunk, scale):
    """T <= 2 H or one chunk takes the single piece, (257, 128) the chunked form.  d(logits) are rounded to bf16 (2^-9) and
    gradients once more, so 2^-7 of the norm bounds both."""
    gen = torch.Generator().manual_seed(T)
    h0, w0 = torch.randn(T, H, generator=gen).to(torch.bfloat16), (torch.randn(V, H, generator=gen) * H ** -0.5).to(torch.bfloat16)
    lab = torch.randint(0, V, (T,), generator=gen)
    lab[::5] = -100
    h, w = h0.cuda().requires_grad_(True), w0.cuda().requires_grad_(True)
    loss = ops.linear_cross_entropy(h, w, lab.cuda(), chunk_size=chunk) * scale
    loss.backward(retain_graph=True)
    first = h.grad.clone(), w.grad.clone()
    h.grad = w.grad = None
    loss.backward()                                   # the saved pieces survive a second backward
    assert torch.equal(h.grad, first[0]) and torch.equal(w.grad, first[1])
    hd, wd = h0.double().requires_grad_(True), w0.double().requires_grad_(True)
    want = torch.nn.functional.cross_entropy(hd @ wd.t(), lab, ignore_index=-100, reduction="sum") * scale
    if (lab >= 0).any():
        want.backward()
    else:
        want, hd.grad, wd.grad = torch.zeros(()), torch.zeros_like(hd), torch.zeros_like(wd)
    assert abs(loss.item() - want.item()) <= 2e-3 * max(1.0, abs(want.item()))
    for a, b in ((h.grad, hd.grad), (w.grad, wd.grad)):
        assert (a.cpu().double() - b).norm() <= 2 ** -7 * b.norm() + 1e-12, ((a.cpu().double() - b).norm() / b.norm())


@pytest.mark.gpu
@pytest.mark.parametrize("M, N, K, out_dtype, accumulate", [(1, 8, 8, torch.bfloat16, False), (200, 264, 72, torch.float32, False),
                                                            (129, 40, 64, torch.float32, True), (256, 512, 128, torch.bfloat16, True)])
def test_scaled_store_multiplies_the_product_only(M, N, K, out_dtype, accumulate):
    from torchturbo_b200 import kernels as KN

    torch.manual_seed(M)
    a, b = (torch.randn(s, K, device="cuda").to(torch.bfloat16) for s in (M, N))
    alpha = torch.tensor([-0.75], device="cuda")
    base = torch.randn(M, N, device="cuda").to(out_dtype)
    out = base.clone()
    KN.gemm(a, b, out=out, accumulate=accumulate, alpha=alpha)
    want = -0.75 * (a.double() @ b.double().t()) + (base.double() if accumulate else 0.0)
    tol = 2 ** -8 if out_dtype == torch.bfloat16 else 1e-5
    assert (out.double() - want).abs().max() <= tol * want.abs().max()
