"""The row-marching 3x3 convolution against im2col + GEMM on the same inputs:
both accumulate the same BF16 products in the same order, so the results are
the same bits.  Sizes: one row and one tile, ragged widths (a second, nearly
empty strip), chunks of one and of many rows, output widths that are no
multiple of the tile, FP32 and BF16 stores."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(Bn, H, W, C, N):
    g = torch.Generator(device="cuda").manual_seed(Bn + H + W + C + N)
    x = torch.randn(Bn, H, W, C, generator=g, device="cuda").to(torch.bfloat16)
    Wb = (torch.randn(N, 9 * C, generator=g, device="cuda") * 0.1).to(torch.bfloat16)
    return x, Wb, torch.randn(N, generator=g, device="cuda")


@pytest.mark.parametrize("Bn,H,W,C,N,out_mode", [
    (1, 1, 64, 8, 32, 1), (2, 9, 129, 8, 32, 1), (1, 300, 257, 8, 40, 0), (2, 7, 130, 32, 32, 1),
    (1, 700, 128, 32, 64, 1), (3, 33, 70, 16, 5, 0), (1, 40, 200, 96, 32, 1), (1, 30, 256, 64, 64, 1),
    (1, 21, 128, 192, 64, 0), (2, 17, 127, 128, 128, 1)])
def test_conv_rows_equals_im2col_gemm(Bn, H, W, C, N, out_mode):
    from glide_b200.guess import _err_flag, conv3x3, gemm, im2col3
    x, Wb, bias = _inputs(Bn, H, W, C, N)
    dt = torch.bfloat16 if out_mode == 1 else torch.float32
    a = torch.empty((Bn * H * W, N), dtype=dt, device="cuda")
    b = torch.full_like(a, float("nan"))
    gemm(im2col3(x), Wb, a, bias=bias, relu=True, out_mode=out_mode)
    conv3x3(x, Wb, b, bias=bias, relu=True, out_mode=out_mode)
    torch.cuda.synchronize()
    assert int(_err_flag(x.device).item()) == 0
    assert torch.equal(a, b)
