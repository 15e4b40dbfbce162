"""Products cut along K: the rule, and values at the edges of tiles, pieces and k-blocks."""
import pytest
import torch


def test_rule_cuts_long_products_with_few_tiles_only():
    from torchturbo_b200.kernels import gemm_splits

    assert gemm_splits(4096, 4096, 4096, 148) == 1            # every SM has a tile
    assert gemm_splits(300, 512, 512, 148) == 1               # short K
    assert gemm_splits(300, 512, 32000, 148) == 15            # 6 tiles, 500 k-blocks: 32 or more a piece
    assert gemm_splits(1024, 2048, 151936, 148) == 2          # 64 tiles
    assert gemm_splits(1280, 2048, 151936, 148) == 1          # 80 tiles: more than half of the SMs
    assert gemm_splits(128, 128, 6208, 148) == 3              # 97 k-blocks: 33, 33, 31
    assert gemm_splits(1, 8, 4095, 148) == 2 and gemm_splits(1, 12, 65536, 148) == 1 and gemm_splits(0, 8, 65536, 148) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("M, N, K", [(1, 8, 4096), (129, 264, 4104), (300, 512, 32000), (128, 128, 6208), (64, 1024, 12352)])
@pytest.mark.parametrize("a_mn, b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("mode", ["bf16", "fp32", "accumulate", "accumulate_bf16", "residual", "alpha", "alpha_accumulate"])
def test_split_products(M, N, K, a_mn, b_mn, mode):
    """fp32 accumulation of bf16 products in another order: 1e-5 of the largest value; a bf16 result adds its rounding."""
    from torchturbo_b200 import kernels as KN

    if a_mn and M % 8:
        M += 8 - M % 8                                         # rows of the MN-major operand start on 16 bytes
    torch.manual_seed(K)
    a, b = (torch.randn(s, K, device="cuda").to(torch.bfloat16) for s in (M, N))
    want = a.double() @ b.double().t()
    A = a.t().contiguous() if a_mn else a
    B = b.t().contiguous() if b_mn else b
    assert KN.gemm_splits(M, N, K, KN.num_sms()) > 1
    if mode == "accumulate":
        out = torch.randn(M, N, device="cuda")
        want = want + out.double()
        got = KN.gemm(A, B, a_mn=a_mn, b_mn=b_mn, out=out, accumulate=True)
    elif mode == "accumulate_bf16":
        out = torch.randn(M, N, device="cuda").to(torch.bfloat16)
        want = want + out.double()
        got = KN.gemm(A, B, a_mn=a_mn, b_mn=b_mn, out=out, accumulate=True)
    elif mode.startswith("alpha"):                             # scales the product, not what it is added to
        out = torch.randn(M, N, device="cuda") if mode == "alpha_accumulate" else None
        want = -0.75 * want + (out.double() if out is not None else 0.0)
        got = KN.gemm(A, B, a_mn=a_mn, b_mn=b_mn, out=out, accumulate=out is not None, alpha=torch.tensor([-0.75], device="cuda"))
    elif mode == "residual":
        res = torch.randn(M, N, device="cuda").to(torch.bfloat16)
        want = want + res.double()
        got = KN.gemm(A, B, a_mn=a_mn, b_mn=b_mn, residual=res)
    else:
        got = KN.gemm(A, B, a_mn=a_mn, b_mn=b_mn, out_dtype=torch.float32 if mode == "fp32" else torch.bfloat16)
    tol = 1e-5 if got.dtype == torch.float32 else 2 ** -8
    assert (got.double() - want).abs().max() <= tol * want.abs().max()
    assert KN.status() == (0, 0)
