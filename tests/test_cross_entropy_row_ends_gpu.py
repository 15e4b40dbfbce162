"""Cross entropy with its gradient in place at row lengths around a block's stride, against float64."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [8, 8184, 8192, 8200, 16384, 16392, 40968])
def test_row_ends(V, in_place=True):
    from torchturbo_b200 import kernels as K

    g = torch.Generator().manual_seed(V)
    x = (torch.randn(5, V, generator=g) * 3).bfloat16()
    labels = torch.tensor([0, V - 1, V // 2, -100, V - 8])
    ref = x.double()
    p = torch.softmax(ref, -1)
    lse = torch.logsumexp(ref, -1)
    valid = labels >= 0
    loss = torch.where(valid, lse - ref.gather(1, labels.clamp(min=0)[:, None])[:, 0], torch.zeros(()).double())
    grad = p.clone()
    grad[torch.arange(5), labels.clamp(min=0)] -= 1
    grad[~valid] = 0
    dev = x.cuda()
    out = dev if in_place else torch.empty_like(dev)
    got = K.cross_entropy(dev, labels.cuda(), grad_out=out)
    # the sum's and the exponentials' fp32 errors, some 2^-20 of a probability and of the loss's operands; the gradient is rounded to
    # bf16 (8 significant bits, at most 2^-8 of a value)
    assert ((got.double().cpu() - loss).abs() <= (lse.abs() + ref.abs().amax(1)) * 2.0 ** -19).all()
    assert ((out.double().cpu() - grad).abs() <= grad.abs() * 2.0 ** -8 + p * 2.0 ** -17 + 1e-37).all()


@pytest.mark.parametrize("V, in_place", [(83992, False), (84000, False), (98312, False), (113992, True), (114000, True), (122888, True)])
def test_row_ends_at_the_order_of_the_second_pass(V, in_place):
    test_row_ends(V, in_place)
