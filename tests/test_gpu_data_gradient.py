"""Data gradient of the training layer: every tap's sum over the output
channels is an FP32 number of its own and the nine are added tap after tap, as
col2im adds the product of gz and the transposed weights.  The same bits as
that pair, at ragged pixel counts, channel tiles and output widths (multiples
of 16 in one kernel, others by GEMM and col2im)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Bn,H,W,Cin,Cout", [(1, 1, 3, 8, 16), (2, 9, 13, 40, 48), (1, 20, 66, 64, 128), (2, 8, 32, 192, 256),
                                             (3, 30, 128, 32, 32), (1, 7, 384, 16, 96), (2, 5, 37, 72, 24)])
def test_data_gradient_adds_the_taps_in_order(Bn, H, W, Cin, Cout):
    from glide_b200.guess import Conv3x3ReLU, _err_flag, col2im3, gemm, transpose
    g = torch.Generator(device="cuda").manual_seed(H + W + Cin + Cout)
    x = torch.randn(Bn, H, W, Cin, generator=g, device="cuda").to(torch.bfloat16).requires_grad_()
    Wf = torch.randn(Cout, 9 * Cin, generator=g, device="cuda") * 0.1
    b = torch.randn(Cout, generator=g, device="cuda")
    y = Conv3x3ReLU.apply(x, Wf, b, True)
    gy = torch.randn(Bn, H, W, Cout, generator=g, device="cuda").to(torch.bfloat16)
    dx, = torch.autograd.grad(y, x, gy)
    gz = (gy * (y > 0)).reshape(-1, Cout)
    dcol = torch.empty(Bn * H * W, 9 * Cin, device="cuda")
    gemm(gz, transpose(Wf.to(torch.bfloat16)), dcol, out_mode=0)
    assert torch.equal(dx, col2im3(dcol, (Bn, H, W, Cin)).to(torch.bfloat16))
    assert int(_err_flag(x.device).item()) == 0


@pytest.mark.parametrize("which", ["x", "gy", "y"])
def test_training_layer_takes_unaligned_slices(which):
    """Inputs and gradients that start off a 16-byte boundary (a slice of a flat
    buffer) give the bits of aligned copies."""
    from glide_b200.guess import Conv3x3ReLU
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(1, 9, 20, 16, generator=g, device="cuda").to(torch.bfloat16)
    Wf, b = torch.randn(32, 9 * 16, generator=g, device="cuda") * 0.1, torch.randn(32, generator=g, device="cuda")
    gy = torch.randn(1, 9, 20, 32, generator=g, device="cuda").to(torch.bfloat16)

    def shifted(t):
        s = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].view(t.shape)
        return s.copy_(t)

    def run(x, gy):
        x, W, bb = x.detach().requires_grad_(), Wf.clone().requires_grad_(), b.clone().requires_grad_()
        y = Conv3x3ReLU.apply(x, W, bb, True)
        if which == "y":   # a hook may keep what is saved for backward anywhere
            with torch.autograd.graph.saved_tensors_hooks(lambda t: t, shifted):
                y = Conv3x3ReLU.apply(x, W, bb, True)
        return [y.detach(), *torch.autograd.grad(y, (x, W, bb), gy)]

    ref = run(x, gy)
    got = run(shifted(x) if which == "x" else x, shifted(gy) if which == "gy" else gy)
    assert all(torch.equal(p, q) for p, q in zip(got, ref))


def test_input_buffer_may_be_refilled_before_backward():
    """The weight gradient belongs to the input of the forward pass, also when
    the caller has put the next batch into the same buffer since."""
    from glide_b200.guess import Conv3x3ReLU
    g = torch.Generator(device="cuda").manual_seed(6)
    x = torch.randn(2, 8, 16, 8, generator=g, device="cuda").to(torch.bfloat16)
    b, gy = torch.zeros(16, device="cuda"), torch.ones(2, 8, 16, 16, device="cuda", dtype=torch.bfloat16)
    Wf = (torch.randn(16, 72, generator=g, device="cuda") * 0.1).requires_grad_()
    ref, = torch.autograd.grad(Conv3x3ReLU.apply(x, Wf, b, True), Wf, gy)
    y = Conv3x3ReLU.apply(x, Wf, b, True)
    x.zero_()
    assert torch.equal(torch.autograd.grad(y, Wf, gy)[0], ref)


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_border_pixels_do_not_see_taps_outside(bad):
    """A tap outside the image adds nothing, whatever its weight."""
    from glide_b200.guess import _data_grad, col2im3, gemm, transpose
    g = torch.Generator(device="cuda").manual_seed(3)
    shape, Cout = (2, 5, 7, 8), 16
    W = torch.randn(Cout, 9, 8, generator=g, device="cuda")
    W[3, 0, 2] = bad
    Wb = W.view(Cout, 72).to(torch.bfloat16)
    gz = torch.randn(70, Cout, generator=g, device="cuda").to(torch.bfloat16)
    dx = _data_grad(gz, Wb, shape)
    dcol = torch.empty(70, 72, device="cuda")
    gemm(gz, transpose(Wb), dcol, out_mode=0)
    ref = col2im3(dcol, shape).to(torch.bfloat16)
    assert torch.equal(dx.isnan(), ref.isnan()) and torch.equal(dx[~ref.isnan()], ref[~ref.isnan()])
    assert bool(ref[..., 2].isfinite().any()) and not bool(ref[..., 2].isfinite().all())
