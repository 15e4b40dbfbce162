"""The SwiGLU backward that also returns the activation."""
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("R, F, rows", [(1, 8, 1), (300, 768, 257), (65, 200, 0), (17, 4104, 17)])
def test_activation_from_the_backward_pass_is_the_forward_result(R, F, rows):
    from torchturbo_b200 import kernels as K

    torch.manual_seed(R)
    x = torch.randn(R, 2 * F, device="cuda").to(torch.bfloat16)
    dy = torch.randn(R, F, device="cuda").to(torch.bfloat16)
    sc = torch.rand(R, device="cuda")
    n = torch.tensor([rows], dtype=torch.int32, device="cuda")
    y = torch.full((R, F), 7.0, device="cuda", dtype=torch.bfloat16)
    dx, ds = K.swiglu_bwd(dy, x, sc, want_dscale=True, nrows=n, y_out=y)
    dx2, ds2 = K.swiglu_bwd(dy, x, sc, want_dscale=True)
    want = K.swiglu_fwd(x, sc)
    assert torch.equal(y[:rows], want[:rows]) and bool((y[rows:] == 7).all())      # rows behind the fill stay as they were
    assert torch.equal(dx[:rows], dx2[:rows]) and torch.equal(ds[:rows], ds2[:rows])
