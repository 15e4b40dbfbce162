"""Gates of a gated delta net in one launch each way, and several projections of the same rows, against 64 bits and the operators they
stand for."""
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("T, H", [(1, 1), (7, 31), (300, 33), (4099, 32), (70, 200)])
@pytest.mark.parametrize("dtypes", [(torch.bfloat16, torch.bfloat16), (torch.float32, torch.bfloat16), (torch.float32, torch.float32)])
def test_gates(T, H, dtypes):
    from torchturbo_b200.ops import ops

    gen = torch.Generator("cuda").manual_seed(T)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)      # noqa: E731
    ab = (rnd(T, 2 * H) * 8).bfloat16()                        # beyond the threshold of the softplus; columns of one matrix
    ab[0, 0] = 30.0
    a, b = (t.requires_grad_() for t in ab.split(H, 1))
    A, dt = rnd(H).to(dtypes[0]).requires_grad_(), rnd(H).to(dtypes[1]).requires_grad_()
    d = rnd(T, H), rnd(T, H)
    g, beta = ops.gdn_gates(a, b, A, dt)
    grads = torch.autograd.grad((g, beta), (a, b, A, dt), d)
    A64, dt64, a64, b64 = (t.detach().double().requires_grad_() for t in (A, dt, a, b))
    want = -A64.exp() * torch.nn.functional.softplus(a64 + dt64), torch.sigmoid(b64)
    for x, y in zip((g, beta), want):
        assert ((x.double() - y).abs() <= y.abs() * 2.0 ** -20 + 2.0 ** -24).all()      # a handful of fp32 functions and roundings
    exact = torch.autograd.grad(want, (a64, b64, A64, dt64), [t.double() for t in d])
    size = [t.abs() for t in exact[:2]] + [(d[0].double() * want[0]).abs().sum(0), exact[0].abs().sum(0)]
    near_one = d[1].double().abs() * 2.0 ** -23              # of 1 - sigmoid where the fp32 sigmoid is close to one
    for x, y, m, more in zip(grads, exact, size, (0.0, near_one, 0.0, 0.0)):
        unit = 2.0 ** -8 if x.dtype == torch.bfloat16 else 0.0
        assert ((x.double() - y).abs() <= y.abs() * unit + m * 2.0 ** -16 + more + 1e-7).all()
    again = torch.autograd.grad(ops.gdn_gates(a, b, A, dt), (a, b, A, dt), [t.clone().requires_grad_() for t in d], create_graph=True)
    for x, y in zip(again, grads):
        assert torch.allclose(x.float(), y.float(), rtol=2.0 ** -7, atol=1e-4)
    assert again[0].requires_grad


@pytest.mark.gpu
@pytest.mark.parametrize("T", [1, 130, 1000])
@pytest.mark.parametrize("widths", [(256, 128, 32, 32), (64, 8), (512,), (8, 264, 16, 64, 72)])
def test_linears(T, widths):
    from torchturbo_b200.ops import ops

    gen = torch.Generator("cuda").manual_seed(T)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen).bfloat16()      # noqa: E731
    x, ws, dys = rnd(T, 192).requires_grad_(), [rnd(n, 192).requires_grad_() for n in widths], [rnd(T, n) for n in widths]
    ys = ops.linears(x, *ws)
    got = torch.autograd.grad(ys, (x, *ws), dys)
    for y, w in zip(ys, ws):
        assert torch.equal(y, ops.linear(x, w))
    for g, w, dy in zip(got[1:], ws, dys):
        exact, mag = dy.double().t() @ x.double(), dy.double().abs().t() @ x.double().abs()
        assert ((g.double() - exact).abs() <= exact.abs() * 2.0 ** -8 + mag * 2.0 ** -15).all()
    exact = sum(dy.double() @ w.double() for w, dy in zip(ws, dys))
    mag = sum(dy.double().abs() @ w.double().abs() for w, dy in zip(ws, dys))
    # every product is added in fp32 to what the ones before left in bf16
    part = sum((dy.double() @ w.double()).abs() for w, dy in zip(ws, dys))
    assert ((got[0].double() - exact).abs() <= part * len(ws) * 2.0 ** -8 + mag * 2.0 ** -15).all()


@pytest.mark.gpu
def test_linears_with_gradient_buffers_and_unused_results():
    from torchturbo_b200.ops import ops

    gen = torch.Generator("cuda").manual_seed(0)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen).bfloat16()      # noqa: E731
    x, ws = rnd(200, 128).requires_grad_(), [rnd(n, 128).requires_grad_() for n in (96, 16, 24)]
    ws[1].main_grad = torch.zeros(16, 128, device="cuda")
    dy, y = rnd(200, 16), ops.linears(x, *ws)
    grads = torch.autograd.grad(y[1], (x, *ws), dy, allow_unused=True)
    assert all(g is None for g in grads[1:])
    assert torch.allclose(ws[1].main_grad, dy.float().t() @ x.float(), atol=2e-3)
    assert torch.equal(grads[0], torch.autograd.grad(ops.linear(x, ws[1].detach()), x, dy)[0])
