"""Multi-tensor AdamW at the edges of its chunks: every element is updated once, whatever the tensor sizes."""
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [[1], [16383], [16384], [16385, 3, 40000], [5, 16384 * 3 + 1, 1, 7]])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_every_element_moves_as_on_the_cpu(sizes, dtype):
    """Same fp32 formulas on both sides; the GPU contracts products and divides approximately: a few units of 2^-23."""
    from torchturbo_b200.engine.optimizers.fused_adamw import FusedAdamW

    gen = torch.Generator().manual_seed(sum(sizes))
    start = [torch.randn(n, generator=gen).to(dtype) for n in sizes]
    grads = [[torch.randn(n, generator=gen).to(dtype) for n in sizes] for _ in range(2)]
    res, norms = [], []
    for dev in ("cuda", "cpu"):
        ps = [torch.nn.Parameter(t.to(dev, copy=True)) for t in start]
        opt = FusedAdamW(ps, lr=1e-2, betas=(0.9, 0.95), weight_decay=0.1)
        for step in grads:
            for p, g in zip(ps, step):
                p.grad = g.to(dev, copy=True)
            if dev == "cuda":
                norms.append(opt.grad_sq_sum().item())
            opt.set_clip_coef(torch.tensor(0.5, device=dev))
            opt.step()
        res.append([opt.state[p].get("master", p.detach()).float().cpu() for p in ps] + [opt.state[p]["exp_avg_sq"].cpu() for p in ps])
    for a, b in zip(*res):
        assert torch.allclose(a, b, rtol=1e-5, atol=1e-6)
    for got, step in zip(norms, grads):
        want = sum(g.double().square().sum().item() for g in step)
        assert abs(got - want) <= 1e-5 * want
