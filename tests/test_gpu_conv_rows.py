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
    (1, 21, 128, 192, 64, 0), (2, 17, 127, 128, 128, 1), (1, 9, 100, 256, 256, 1), (2, 5, 37, 72, 96, 0)])
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


@pytest.mark.parametrize("Bn,H,W,C0,C1,N", [(1, 2, 128, 64, 32, 32), (2, 34, 130, 128, 64, 64), (1, 16, 66, 256, 128, 128),
                                            (2, 6, 10, 8, 16, 24)])
def test_two_source_conv_equals_joined(Bn, H, W, C0, C1, N):
    """Upsampling and concatenation read inside the convolution: the same bits
    as on the joined tensor (row march, specialised GEMM, narrow images)."""
    from glide_b200.guess import _up, conv3x3_relu, conv3x3_up_cat
    g = torch.Generator(device="cuda").manual_seed(H + W + C0)
    x = torch.randn(Bn, H // 2, W // 2, C0, generator=g, device="cuda").to(torch.bfloat16)
    skip = torch.randn(Bn, H, W, C1, generator=g, device="cuda").to(torch.bfloat16)
    Wf = torch.randn(N, 9 * (C0 + C1), generator=g, device="cuda") * 0.1
    b = torch.randn(N, generator=g, device="cuda")
    ref = conv3x3_relu(torch.cat([_up(x), skip], dim=3), Wf, b)
    assert torch.equal(conv3x3_up_cat(x, skip, Wf, b), ref)


@pytest.mark.parametrize("shape", [(1, 2, 2, 8), (2, 34, 50, 32), (1, 16, 66, 64)])
def test_pool_equals_mean(shape):
    """One-pass pooling against the torch expression (the sums of four BF16
    values differ by an FP32 rounding at most, i.e. by at most one BF16 step)."""
    from glide_b200.guess import _pool
    g = torch.Generator(device="cuda").manual_seed(shape[1])
    x = torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16)
    Bn, H, W, Cc = shape
    ref = x.view(Bn, H // 2, 2, W // 2, 2, Cc).float().mean((2, 4))
    assert (_pool(x).float() - ref).abs().max().item() <= 2.0 ** -8 * ref.abs().max().item()


@pytest.mark.parametrize("Bn,H,W,C,N", [(1, 1, 3, 8, 8), (2, 9, 13, 40, 24), (1, 16, 16, 32, 136), (3, 20, 37, 64, 64),
                                         (2, 3, 128, 32, 32), (1, 7, 384, 40, 24), (3, 8, 32, 96, 160)])
def test_weight_gradient_equals_transposed_gemm(Bn, H, W, C, N):
    """Pixels as the contraction, read in place: the same bits as the GEMM on
    the transposes of gz and of the im2col matrix (ragged pixel count and
    channel tiles, more than 128 output channels)."""
    from glide_b200 import _native as NT
    from glide_b200.guess import _err_flag, _lib, gemm, im2col3, transpose
    g = torch.Generator(device="cuda").manual_seed(H + W + C + N)
    x = torch.randn(Bn, H, W, C, generator=g, device="cuda").to(torch.bfloat16)
    gz = torch.randn(Bn * H * W, N, generator=g, device="cuda").to(torch.bfloat16)
    P = Bn * H * W
    # the pixel count padded to a multiple of 8 with zero rows keeps the GEMM on its aligned kernel
    pad = (-P) % 8
    zp, cp = (torch.cat([t, t.new_zeros(pad, t.shape[1])]) for t in (gz, im2col3(x)))
    ref = torch.empty(N, 9 * C, device="cuda")
    gemm(transpose(zp), transpose(cp), ref)
    out = torch.full_like(ref, float("nan"))
    NT.check(_lib().glide_conv3x3_wgrad_bf16(gz.data_ptr(), x.data_ptr(), out.data_ptr(), Bn, H, W, C, N,
                                             _err_flag(x.device).data_ptr(), NT.stream_handle()), "wgrad")
    torch.cuda.synchronize()
    assert int(_err_flag(x.device).item()) == 0
    assert torch.equal(out, ref)


@pytest.mark.parametrize("P,N,relu", [(1, 8, True), (1000, 24, True), (70000, 256, True), (333, 32, False)])
def test_relu_gradient_and_bias_sum(P, N, relu):
    """gz exactly; db within FP32 summation error, P eps of the sum of |gz|
    (each block adds at most P values in FP32)."""
    from glide_b200.guess import _relu_grad
    g = torch.Generator(device="cuda").manual_seed(P)
    gy = torch.randn(P, N, generator=g, device="cuda").to(torch.bfloat16)
    y = torch.relu(torch.randn(P, N, generator=g, device="cuda")).to(torch.bfloat16)
    gz, db = _relu_grad(gy, y, relu)
    ref = gy.float() * (y > 0) if relu else gy.float()
    assert torch.equal(gz.float(), ref)
    err = (db.double() - ref.double().sum(0)).abs()
    assert bool((err <= min(P, 4096) * 6e-8 * ref.double().abs().sum(0) + 1e-30).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_features_equal_torch(dtype):
    """One-pass network input = the torch expression, bit for bit (values over
    the geometry's ranges, beta down to 0 and below the clamp, infinities, NaN)."""
    from glide_b200 import guess
    g = torch.Generator(device="cuda").manual_seed(3)
    f = [torch.randn(1, 211, 307, generator=g, device="cuda", dtype=torch.float64) * s for s in (1500.0, 600.0, 1.0, 40.0)]
    f[2] = torch.exp(3 * f[2]) * 0.1
    f[2].view(-1)[:5] = torch.tensor([0.0, -1.0, 1e-9, float("inf"), float("nan")], device="cuda")
    f[0].view(-1)[:2] = torch.tensor([float("inf"), float("nan")], device="cuda")
    f = [t.to(dtype) for t in f]
    one = guess.features(*f)
    ref = guess.features(*(t.transpose(1, 2).contiguous().transpose(1, 2) for t in f))   # not contiguous: torch path
    same = (one == ref) | (one.isnan() & ref.isnan())
    assert bool(same.all())


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 40, 33), (3, 17, 70)])
def test_faces_equal_torch(shape):
    from glide_b200 import guess

    class Fixed(torch.nn.Module):
        def __init__(self, p):
            super().__init__()
            self.p = p

        def forward(self, x):
            return self.p

    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    p = torch.randn(*shape, 2, generator=g, device="cuda")
    z = torch.ones(shape, device="cuda")
    u, v = guess.GuessModel(Fixed(p)).predict(z, z, z, z)
    ru, rv = guess.faces_from_cells(p)
    if shape[0] == 1:
        ru, rv = ru[0], rv[0]
    assert torch.equal(u, ru.double()) and torch.equal(v, rv.double())


@pytest.mark.parametrize("C,C1,N,W", [(8, 0, 32, 64), (32, 0, 40, 130), (64, 32, 32, 70), (128, 64, 64, 128)])
def test_fp32_weights_equal_cast_weights(C, C1, N, W):
    """Weights rounded while staged = weights cast to BF16 before."""
    from glide_b200.guess import _rows_f32w, _up, conv3x3
    g = torch.Generator(device="cuda").manual_seed(C + N)
    up = 1 if C1 else 0
    x = torch.randn(2, 6 >> up, W >> up, C, generator=g, device="cuda").to(torch.bfloat16)
    skip = torch.randn(2, 6, W, C1, generator=g, device="cuda").to(torch.bfloat16) if C1 else None
    Wf, b = torch.randn(N, 9 * (C + C1), generator=g, device="cuda"), torch.randn(N, generator=g, device="cuda")
    y = torch.empty(2, 6, W, N, dtype=torch.bfloat16, device="cuda")
    assert _rows_f32w(x, up, skip, Wf, b, True, y)
    ref = torch.empty(2 * 6 * W, N, dtype=torch.bfloat16, device="cuda")
    conv3x3(torch.cat([_up(x), skip], 3).contiguous() if C1 else x, Wf.to(torch.bfloat16), ref, bias=b, relu=True)
    assert torch.equal(y.view(-1, N), ref)
