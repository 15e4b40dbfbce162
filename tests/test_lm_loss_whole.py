"""lm_head + cross entropy in one piece against the chunked accumulation, and the scaled GEMM store it relies on."""
import pytest
import torch

from torchturbo_b200.ops import ops


def _on_cpu(monkeypatch):
    """Torch products in the place of the kernels, unseen by autograd as those are."""
    from torchturbo_b200.ops.providers import b200

    @torch.no_grad()
    def gemm(a, b, *, a_mn=False, b_mn=False, out=None, out_dtype=torch.bfloat16, accumulate=False, alpha=None):
        c = (a.t() if a_mn else a).float() @ (b if b_mn else b.t()).float() * (alpha if alpha is not None else 1.0)
        if out is None:
            return c.to(out_dtype)
        return out.copy_(c + out if accumulate else c)

    def cross_entropy(logits, labels, grad_out=None):
        x = logits.float().requires_grad_(True)
        with torch.enable_grad():
            loss = torch.nn.functional.cross_entropy(x, labels, ignore_index=-100, reduction="none")
            (g,) = torch.autograd.grad(loss.sum(), x)
        if grad_out is not None:
            grad_out.copy_(g)
        return loss.detach()

    monkeypatch.setattr(b200.K, "gemm", gemm)
    monkeypatch.setattr(b200.K, "cross_entropy", cross_entropy)
    return b200.LinearCrossEntropyFn


@pytest.mark.parametrize("T, chunk, held", [
    (16, 4, "logits"), (16, 64, "logits"), (17, 64, "direct"), (17, 17, "direct"), (17, 16, "accumulator"), (17, 4, "accumulator")])
def test_what_is_held_for_the_backward_follows_from_the_rows(T, chunk, held, monkeypatch):
    """H = 8: up to 16 rows d(logits); beyond that d(W), in the weight's dtype from one chunk and in fp32 from several."""
    fn = _on_cpu(monkeypatch)
    torch.manual_seed(T)
    H, V = 8, 24
    h, w = torch.randn(T, H).to(torch.bfloat16).requires_grad_(True), torch.randn(V, H).to(torch.bfloat16).requires_grad_(True)
    lab = torch.randint(0, V, (T,))
    loss = fn.apply(h, w, lab, chunk) * 0.5
    kept = {(tuple(t.shape), t.dtype) for t in loss.grad_fn.next_functions[0][0].saved_tensors if t is not None}
    want = {"logits": {((T, V), torch.bfloat16), ((T, H), torch.bfloat16)}, "direct": {((V, H), torch.bfloat16), ((T, H), torch.bfloat16)},
            "accumulator": {((V, H), torch.float32), ((T, H), torch.bfloat16)}}[held]
    assert kept == want
    loss.backward()
    hd, wd = h.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    torch.nn.functional.cross_entropy(hd @ wd.t(), lab, reduction="sum").mul(0.5).backward()
    for a, b in ((h.grad, hd.grad), (w.grad, wd.grad)):
        assert (a.double() - b).norm() <= 2 ** -6 * b.norm()


@pytest.mark.parametrize("T", [16, 17])
def test_incoming_gradient_stays_in_a_graph_of_the_gradients(T, monkeypatch):
    """d(grad)/d(scale) for a loss that a trainable scale multiplies, in the single piece (16 rows) as in the other forms."""
    fn = _on_cpu(monkeypatch)
    torch.manual_seed(0)
    h, w = torch.randn(T, 8).to(torch.bfloat16).requires_grad_(True), torch.randn(24, 8).to(torch.bfloat16).requires_grad_(True)
    scale, lab = torch.tensor(0.5, requires_grad=True), torch.randint(0, 24, (T,))
    gh, gw = torch.autograd.grad(fn.apply(h, w, lab, 64) * scale, (h, w), create_graph=True)
    for g in (gh, gw):
        (d,) = torch.autograd.grad(g.float().square().sum(), scale, retain_graph=True)
        assert abs(d.item() - 4 * g.float().square().sum().item()) <= 2 ** -5 * abs(d.item())      # grad = scale * x


@pytest.mark.gpu
@pytest.mark.parametrize("T, H, V, chunk", [(1, 64, 128, 4), (130, 128, 1000, 64), (257, 128, 1000, 64), (200, 64, 520, 512), (256, 128, 1032, 100)])
@pytest.mark.parametrize("scale", [1.0, 0.37])
def test_whole_and_chunked_forms_agree_with_fp64(T, H, V, chunk, scale):
    """T <= 2 H takes the single piece, (200, 64) one chunk, (257, 128) several.  d(logits) are rounded to bf16 (2^-9) and
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
