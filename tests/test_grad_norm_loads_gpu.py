"""Squared norms of gradients against a float64 sum: both types, sizes around a load and a chunk, addresses off the 16-byte grid."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shift", [0, 1])
def test_partials(dtype, shift):
    from torchturbo_b200 import kernels as K

    torch.manual_seed(3)
    sizes = [1, 3, 7, 8, 9, 1023, 2048, 8191, 16383, 16384, 16385, 50001]
    ps = [torch.zeros(n, device="cuda") for n in sizes]
    gs = [torch.randn(n + shift, device="cuda").to(dtype)[shift:] for n in sizes]
    plan = K.MultiTensorPlan(ps, [torch.zeros_like(p) for p in ps], [torch.zeros_like(p) for p in ps])
    plan.refresh_grads(gs)
    part = K.grad_sqnorm_partials(plan, 0.5).double().cpu()
    at = 0
    for n, g in zip(sizes, gs):
        chunks = -(-n // K.ADAM_CHUNK)
        want = 0.25 * g.double().square().sum().item()
        # positive terms: each of at most 64 + 12 additions on a term's way (a thread's, the block's) rounds by 2^-24
        assert abs(part[at: at + chunks].sum().item() - want) <= want * 80 * 2.0 ** -24
        at += chunks
    assert at == part.numel()


@pytest.mark.parametrize("n", [1, 255, 257, 64 * 256 + 1, 100000])
def test_copy_words_both_ways(n):
    from torchturbo_b200 import kernels as K

    src = torch.arange(n, dtype=torch.int32).pin_memory()
    dev, back = torch.full((n + 1,), -1, dtype=torch.int32, device="cuda"), torch.full((n,), -1, dtype=torch.int32).pin_memory()
    K.copy_words(dev[:n], src)
    K.copy_words(back, dev[:n])
    torch.cuda.synchronize()
    assert torch.equal(back, src) and dev[n].item() == -1
    with pytest.raises(AssertionError):
        K.copy_words(dev[:n], torch.arange(n, dtype=torch.int32))     # pageable
    with pytest.raises(AssertionError):
        K.copy_words(dev, src)
