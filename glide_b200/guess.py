"""Learned initial guess: a small U-Net on the B200 tensor cores.

Maps cell fields (H, bed, log beta, B) to cell-centred velocities (u, v),
which are averaged onto the staggered faces and handed to
``IcePhysics.forward(guess=...)``; the plain V-cycle always finishes the
solve and drops the guess if the first cycle does not cut the residual by
``guess_min_reduction``.

Network: 4 resolution levels, 32 base channels (32-64-128-256), two 3x3
conv + ReLU per level, 2x average pooling down, nearest upsampling and skip
concatenation up, a 1x1 head to 2 channels.  Activations are NHWC BF16,
weights are kept in FP32 for the optimiser and cast to BF16 for the
products.  Every convolution runs on the tcgen05 tensor cores with FP32
accumulation in TMEM, without an im2col matrix in either direction
(``glide_conv3x3_bf16`` and its ``cat``, ``rows_f32w``, ``dgrad`` and ``wgrad``
forms; widths that are no multiple of 8 run im2col + ``glide_gemm_bf16``); bias and
ReLU are fused into the epilogue.  In inference the decoder's upsampling and
concatenation are read in place and pooling is one pass; in training they and the
optimiser are element-wise torch glue.  This part has no counterpart in the
reference.
"""
from __future__ import annotations

import ctypes as C
import math
import os
from pathlib import Path

import torch
from torch.autograd import forward_ad

from . import _native as N

DEFAULT_WEIGHTS = Path(__file__).resolve().parent / "guess_weights.pt"
VEL_SCALE = 100.0          # m/a
IN_CH = 8                  # 4 physical inputs zero-padded to 8 channels (16-byte rows)


def _lib():
    lib = N.load()
    if not getattr(lib, "_guess_sigs", False):
        lib.glide_gemm_bf16.argtypes = [C.c_void_p, C.c_int, C.c_void_p, C.c_int, C.c_void_p, C.c_int, C.c_int,
                                        C.c_int, C.c_int, C.c_void_p, C.c_int, C.c_int, C.c_void_p, C.c_void_p]
        lib.glide_gemm_bf16.restype = C.c_int
        lib.glide_im2col3_bf16.argtypes = [C.c_void_p, C.c_void_p] + [C.c_int] * 5 + [C.c_void_p]
        lib.glide_im2col3_bf16.restype = C.c_int
        lib.glide_col2im3_f32.argtypes = [C.c_void_p, C.c_void_p] + [C.c_int] * 5 + [C.c_void_p]
        lib.glide_col2im3_f32.restype = C.c_int
        lib.glide_transpose_bf16.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_int, C.c_void_p]
        lib.glide_transpose_bf16.restype = C.c_int
        lib.glide_conv3x3_bf16.argtypes = [C.c_void_p] + [C.c_int] * 4 + [C.c_void_p, C.c_int, C.c_void_p, C.c_int,
                                                                          C.c_int, C.c_void_p, C.c_int, C.c_int,
                                                                          C.c_void_p, C.c_void_p]
        lib.glide_conv3x3_bf16.restype = C.c_int
        lib.glide_conv3x3_cat_bf16.argtypes = ([C.c_void_p, C.c_int, C.c_int, C.c_void_p] + [C.c_int] * 4 +
                                               [C.c_void_p, C.c_int, C.c_void_p, C.c_int, C.c_int, C.c_void_p,
                                                C.c_int, C.c_int, C.c_void_p, C.c_void_p])
        lib.glide_conv3x3_cat_bf16.restype = C.c_int
        lib.glide_pool2_bf16.argtypes = [C.c_void_p, C.c_void_p] + [C.c_int] * 4 + [C.c_void_p]
        lib.glide_pool2_bf16.restype = C.c_int
        lib.glide_conv3x3_wgrad_bf16.argtypes = [C.c_void_p] * 3 + [C.c_int] * 5 + [C.c_void_p, C.c_void_p]
        lib.glide_conv3x3_wgrad_bf16.restype = C.c_int
        lib.glide_conv3x3_dgrad_bf16.argtypes = [C.c_void_p] * 3 + [C.c_int] * 5 + [C.c_void_p, C.c_void_p]
        lib.glide_conv3x3_dgrad_bf16.restype = C.c_int
        lib.glide_relu_grad_bf16.argtypes = [C.c_void_p] * 5 + [C.c_int64, C.c_int, C.c_int, C.c_void_p]
        lib.glide_relu_grad_bf16.restype = C.c_int
        lib.glide_relu_grad_blocks.argtypes = [C.c_int64, C.c_int]
        lib.glide_relu_grad_blocks.restype = C.c_int
        lib.glide_conv3x3_rows_ok.argtypes = [C.c_int] * 5
        lib.glide_conv3x3_rows_ok.restype = C.c_int
        lib.glide_conv3x3_rows_f32w.argtypes = ([C.c_void_p, C.c_int, C.c_int, C.c_void_p] + [C.c_int] * 4 +
                                                [C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_int, C.c_void_p,
                                                 C.c_void_p])
        lib.glide_conv3x3_rows_f32w.restype = C.c_int
        lib.glide_guess_features.argtypes = [C.c_int] + [C.c_void_p] * 5 + [C.c_int64, C.c_void_p]
        lib.glide_guess_features.restype = C.c_int
        lib.glide_guess_faces.argtypes = [C.c_void_p] * 3 + [C.c_int] * 3 + [C.c_double, C.c_void_p]
        lib.glide_guess_faces.restype = C.c_int
        lib._guess_sigs = True
    return lib


_ERR = {}


def _err_flag(device):
    t = _ERR.get(device)
    if t is None:
        t = torch.zeros(1, dtype=torch.int32, device=device)
        _ERR[device] = t
    return t


def gemm(A, B, out, bias=None, relu=False, out_mode=0):
    """out (+)= A @ B.T on the tensor cores (A: M x K, B: N x K, both BF16)."""
    assert A.dtype == torch.bfloat16 and B.dtype == torch.bfloat16
    assert A.is_contiguous() and B.is_contiguous() and out.is_contiguous()
    M, K = A.shape
    Nn = B.shape[0]
    rc = _lib().glide_gemm_bf16(A.data_ptr(), K, B.data_ptr(), K, out.data_ptr(), Nn, M, Nn, K,
                                None if bias is None else bias.data_ptr(), int(relu), int(out_mode),
                                _err_flag(A.device).data_ptr(), N.stream_handle())
    N.check(rc, "tensor-core gemm")
    return out


def conv3x3(x, Wb, out, bias=None, relu=False, out_mode=1):
    """out (+)= conv3x3(x) on the tensor cores as an implicit GEMM (no im2col
    buffer): x NHWC BF16 with C % 8 == 0, Wb (Cout, 9C) BF16."""
    assert x.dtype == torch.bfloat16 and Wb.dtype == torch.bfloat16
    assert x.is_contiguous() and Wb.is_contiguous() and out.is_contiguous()
    Bn, H, W, Cc = x.shape
    Nn = Wb.shape[0]
    rc = _lib().glide_conv3x3_bf16(x.data_ptr(), Bn, H, W, Cc, Wb.data_ptr(), Wb.shape[1], out.data_ptr(), Nn, Nn,
                                   None if bias is None else bias.data_ptr(), int(relu), int(out_mode),
                                   _err_flag(x.device).data_ptr(), N.stream_handle())
    N.check(rc, "tensor-core conv3x3")
    return out


def im2col3(x):
    Bn, H, W, Cc = x.shape
    col = torch.empty((Bn * H * W, 9 * Cc), dtype=torch.bfloat16, device=x.device)
    N.check(_lib().glide_im2col3_bf16(x.data_ptr(), col.data_ptr(), Bn, H, W, Cc, 9 * Cc, N.stream_handle()),
            "im2col")
    return col


def col2im3(dcol, shape):
    Bn, H, W, Cc = shape
    dx = torch.empty((Bn, H, W, Cc), dtype=torch.float32, device=dcol.device)
    N.check(_lib().glide_col2im3_f32(dcol.data_ptr(), dx.data_ptr(), Bn, H, W, Cc, 9 * Cc, N.stream_handle()),
            "col2im")
    return dx


def transpose(x):
    R, Cc = x.shape
    y = torch.empty((Cc, R), dtype=torch.bfloat16, device=x.device)
    N.check(_lib().glide_transpose_bf16(x.data_ptr(), y.data_ptr(), R, Cc, N.stream_handle()), "transpose")
    return y


def conv3x3_relu(x, W, b, relu=True):
    """relu(conv3x3(x, W) + b).  With autograd recording (training) this is
    Conv3x3ReLU, which keeps x for the weight gradient; without (inference) the
    weights are rounded inside the kernel where the row march takes the shape, with
    a bit-identical result."""
    Bn, H, Wd, Cin = x.shape
    if (torch.is_grad_enabled() and (x.requires_grad or W.requires_grad or b.requires_grad)) or Cin % 8 != 0:
        return Conv3x3ReLU.apply(x, W, b, relu)
    Cout = W.shape[0]
    y = torch.empty((Bn, H, Wd, Cout), dtype=torch.bfloat16, device=x.device)
    x = x.contiguous()
    if not _rows_f32w(x, 0, None, W, b, relu, y):
        conv3x3(x, W.detach().to(torch.bfloat16).contiguous(), y.view(-1, Cout), bias=b.detach(),
                relu=relu, out_mode=1)
    return y


def _rows_f32w(x, up, skip, W, b, relu, y):
    """y = relu(conv3x3(x | skip)) with the FP32 weights rounded inside the
    kernel, where the row march takes the shape; False where it does not.  The
    entry point sees addresses only: types, the weights' width (it assumes
    9 Cin) and the bias are checked here, and what does not fit is left to
    conv3x3, which refuses it or takes its pitch."""
    lib = _lib()
    Bn, H, Wd, Cout = y.shape
    C0, C1 = x.shape[3], 0 if skip is None else skip.shape[3]
    w = W.data_ptr()
    if x.dtype is not torch.bfloat16 or (C1 and skip.dtype is not torch.bfloat16) or \
            W.dtype is not torch.float32 or W.shape != (Cout, 9 * (C0 + C1)) or w % 16 or not W.is_contiguous() or \
            b.dtype is not torch.float32 or b.numel() < Cout or not b.is_contiguous() or \
            not lib.glide_conv3x3_rows_ok(C0, up, C1, Wd, Cout):
        return False
    N.check(lib.glide_conv3x3_rows_f32w(x.data_ptr(), C0, up, skip.data_ptr() if C1 else None, C1, Bn, H, Wd, w,
                                        y.data_ptr(), Cout, b.data_ptr(), int(relu), _err_flag(x.device).data_ptr(),
                                        N.stream_handle()), "tensor-core conv3x3")
    return True


def _in_place(x, skip, W):
    """Whether the two sources can be read as they are: BF16, skip at twice the
    resolution of x, 16-byte aligned channels in both, weights without padding."""
    if x.dtype is not torch.bfloat16 or skip.dtype is not torch.bfloat16 or x.dim() != 4 or skip.dim() != 4:
        return False
    n, h, w, c0 = x.shape
    m, H, Wd, c1 = skip.shape
    return m == n and H == 2 * h and Wd == 2 * w and n * h * w * c0 * c1 > 0 and c0 % 8 == 0 and c1 % 8 == 0 and \
        W.dim() == 2 and W.shape[1] == 9 * (c0 + c1) and x.device == skip.device and \
        (x.data_ptr() | skip.data_ptr() | W.data_ptr()) % 16 == 0


def conv3x3_up_cat(x, skip, W, b):
    """conv3x3_relu(cat([_up(x), skip]), W, b).  Without autograd recording the
    convolution reads both tensors directly where it can (bit-identical); what
    does not fit is joined first, so that torch.cat refuses what it refuses."""
    if not (torch.is_grad_enabled() and any(t.requires_grad for t in (x, skip, W, b))):
        x, skip = x.contiguous(), skip.contiguous()
        if _in_place(x, skip, W):
            return _conv_two_sources(x, skip, W, b)
    return conv3x3_relu(torch.cat([_up(x), skip], dim=3), W, b)


def _conv_two_sources(x, skip, W, b):
    Bn, H, Wd, C1 = skip.shape
    y = torch.empty((Bn, H, Wd, W.shape[0]), dtype=torch.bfloat16, device=x.device)
    if _rows_f32w(x, 1, skip, W, b, True, y):
        return y
    Wb = W.detach().to(torch.bfloat16).contiguous()
    rc = _lib().glide_conv3x3_cat_bf16(x.data_ptr(), x.shape[3], 1, skip.data_ptr(), C1, Bn, H, Wd, Wb.data_ptr(),
                                       Wb.shape[1], y.data_ptr(), y.shape[3], y.shape[3], b.detach().data_ptr(), 1, 1,
                                       _err_flag(x.device).data_ptr(), N.stream_handle())
    N.check(rc, "tensor-core conv3x3 (two sources)")
    return y


def _relu_grad(gy, y, relu):
    """(gz, db): gy masked by y > 0 in BF16 and its channel sums in FP32, one pass."""
    P, Cout = y.shape
    lib = _lib()
    gz = torch.empty_like(y)
    db = torch.empty(Cout, dtype=torch.float32, device=y.device)
    parts = torch.empty(lib.glide_relu_grad_blocks(P, Cout) * Cout, dtype=torch.float32, device=y.device)
    N.check(lib.glide_relu_grad_bf16(gy.data_ptr(), y.data_ptr(), gz.data_ptr(), db.data_ptr(), parts.data_ptr(), P,
                                     Cout, int(relu), N.stream_handle()), "relu gradient")
    return gz, db


def _data_grad(gz, Wb, shape):
    """dx of a 3x3 layer from gz (P, Cout): each tap's sum over Cout in FP32, the
    nine added in FP32.  Output widths that are no multiple of 16 go through
    dcol (P x 9Cin) = gz . W and col2im, the others compute the same numbers in
    one kernel."""
    Bn, H, Wd, Cin = shape
    P, Cout = gz.shape
    Wt = transpose(Wb)
    if Cin % 8 == 0 and Cout % 16 == 0:
        dx = torch.empty(shape, dtype=torch.bfloat16, device=gz.device)
        N.check(_lib().glide_conv3x3_dgrad_bf16(gz.data_ptr(), Wt.data_ptr(), dx.data_ptr(), Bn, H, Wd, Cin, Cout,
                                                _err_flag(gz.device).data_ptr(), N.stream_handle()), "data gradient")
        return dx
    dcol = torch.empty((P, 9 * Cin), dtype=torch.float32, device=gz.device)
    gemm(gz, Wt, dcol, out_mode=0)
    return col2im3(dcol, shape).to(torch.bfloat16)


def _aligned(t):
    """t as the 16-byte loads of the training layer want it: contiguous, copied
    where it starts off a 16-byte boundary."""
    t = t.contiguous()
    return t.clone() if t.data_ptr() % 16 else t


class Conv3x3ReLU(torch.autograd.Function):
    """y = relu(conv3x3(x, W) + b); x NHWC BF16, W (Cout, 9*Cin) FP32 master.

    With Cin and Cout multiples of 8 no im2col matrix exists in the forward
    product and the weight gradient, which gather their shifted pixels
    themselves; the data gradient is _data_grad.  Other widths run im2col +
    GEMM."""

    @staticmethod
    def forward(ctx, x, W, b, relu: bool):
        Bn, H, Wd, Cin = x.shape
        Cout = W.shape[0]
        x = x.contiguous()
        Wb = W.to(torch.bfloat16).contiguous()
        y = torch.empty((Bn * H * Wd, Cout), dtype=torch.bfloat16, device=x.device)
        ctx.implicit = Cin % 8 == 0 and Cout % 8 == 0 and Cout <= 2048
        if ctx.implicit:
            x = _aligned(x)
            conv3x3(x, Wb, y, bias=b, relu=relu, out_mode=1)
            # an input that is not differentiated is often a buffer which the caller fills again
            ctx.save_for_backward(x if ctx.needs_input_grad[0] else x.clone(), Wb, y)
        else:
            col = im2col3(x)
            gemm(col, Wb, y, bias=b, relu=relu, out_mode=1)
            ctx.save_for_backward(col, Wb, y)
        ctx.shape = (Bn, H, Wd, Cin)
        ctx.relu = relu
        return y.view(Bn, H, Wd, Cout)

    @staticmethod
    def backward(ctx, gy):
        src, Wb, y = ctx.saved_tensors
        Bn, H, Wd, Cin = ctx.shape
        Cout = Wb.shape[0]
        P = Bn * H * Wd
        if ctx.implicit:
            src, Wb, y = _aligned(src), _aligned(Wb), _aligned(y.reshape(P, Cout))   # hooks may have moved them
            gz, db = _relu_grad(_aligned(gy.reshape(P, Cout).to(torch.bfloat16)), y, ctx.relu)
            dW = torch.empty((Cout, 9 * Cin), dtype=torch.float32, device=gy.device)
            N.check(_lib().glide_conv3x3_wgrad_bf16(gz.data_ptr(), src.data_ptr(), dW.data_ptr(), Bn, H, Wd, Cin, Cout,
                                                    _err_flag(gy.device).data_ptr(), N.stream_handle()),
                    "weight gradient")
            return _data_grad(gz, Wb, (Bn, H, Wd, Cin)), dW, db, None
        g = gy.reshape(P, Cout).float()
        if ctx.relu:
            g = g * (y > 0)
        gz = g.to(torch.bfloat16).contiguous()
        # weight gradient: dW (Cout x 9Cin) = gz^T (Cout x P) . col (P x 9Cin)
        dW = torch.zeros((Cout, 9 * Cin), dtype=torch.float32, device=gy.device)
        gemm(transpose(gz), transpose(src), dW, out_mode=0)
        db = g.sum(0)
        return _data_grad(gz, Wb, (Bn, H, Wd, Cin)), dW, db, None


class Conv1x1(torch.autograd.Function):
    """Linear head y = x . W^T + b per pixel (x NHWC BF16, y FP32)."""

    @staticmethod
    def forward(ctx, x, W, b):
        Bn, H, Wd, Cin = x.shape
        Cout = W.shape[0]
        xf = x.reshape(-1, Cin).contiguous()
        Wb = W.to(torch.bfloat16).contiguous()
        y = torch.empty((xf.shape[0], Cout), dtype=torch.float32, device=x.device)
        gemm(xf, Wb, y, bias=b, out_mode=0)
        ctx.save_for_backward(xf, Wb)
        ctx.shape = (Bn, H, Wd, Cin)
        return y.view(Bn, H, Wd, Cout)

    @staticmethod
    def backward(ctx, gy):
        xf, Wb = ctx.saved_tensors
        Bn, H, Wd, Cin = ctx.shape
        Cout = Wb.shape[0]
        g = gy.reshape(-1, Cout).float()
        gz = g.to(torch.bfloat16).contiguous()
        dW = torch.zeros((Cout, Cin), dtype=torch.float32, device=gy.device)
        gemm(transpose(gz), transpose(xf), dW, out_mode=0)
        dx = torch.empty((xf.shape[0], Cin), dtype=torch.float32, device=gy.device)
        gemm(gz, transpose(Wb), dx, out_mode=0)
        return dx.view(Bn, H, Wd, Cin).to(torch.bfloat16), dW, g.sum(0)


def _plain(*ts):
    """Whether a kernel may read these tensors by address: ordinary contiguous
    tensors on the current device that nothing differentiates, maps or traces
    (torch's own operations serve all of that)."""
    if torch._C._len_torch_dispatch_stack() or torch.compiler.is_compiling() or torch.jit.is_tracing():
        return False
    dual = forward_ad._current_level >= 0
    return all(t.is_cuda and type(t) in (torch.Tensor, torch.nn.Parameter) and
               not torch._C._functorch.is_functorch_wrapped_tensor(t) and
               t.layout is torch.strided and t.is_contiguous() and t.numel() > 0 and not t.is_neg() and
               not (t.requires_grad and torch.is_grad_enabled()) and
               not (dual and forward_ad.unpack_dual(t).tangent is not None) and
               t.get_device() == torch.cuda.current_device() for t in ts)


def _pool(x):
    Bn, H, W, Cc = x.shape
    if _plain(x) and x.dtype == torch.bfloat16 and Cc % 8 == 0 and H % 2 == 0 and W % 2 == 0 and \
            x.data_ptr() % 16 == 0:
        y = torch.empty((Bn, H // 2, W // 2, Cc), dtype=torch.bfloat16, device=x.device)
        N.check(_lib().glide_pool2_bf16(x.data_ptr(), y.data_ptr(), Bn, H, W, Cc, N.stream_handle()), "pool")
        return y
    return x.view(Bn, H // 2, 2, W // 2, 2, Cc).float().mean((2, 4)).to(torch.bfloat16)


def _up(x):
    return x.repeat_interleave(2, dim=1).repeat_interleave(2, dim=2)


class UNet(torch.nn.Module):
    """4-level, 32-base-channel U-Net (NHWC, BF16 activations)."""

    def __init__(self, base=32, levels=4, in_ch=IN_CH, out_ch=2, seed=0):
        super().__init__()
        g = torch.Generator().manual_seed(seed)
        chans = [base * 2 ** k for k in range(levels)]
        self.levels = levels
        self.ws = torch.nn.ParameterList()
        self.bs = torch.nn.ParameterList()
        self.plan = []   # (cin, cout) of each 3x3 conv, in order

        def add(cin, cout):
            w = torch.randn(cout, 9 * cin, generator=g) * math.sqrt(2.0 / (9 * cin))
            self.ws.append(torch.nn.Parameter(w))
            self.bs.append(torch.nn.Parameter(torch.zeros(cout)))
            self.plan.append((cin, cout))

        cin = in_ch
        for k in range(levels):            # encoder
            add(cin, chans[k])
            add(chans[k], chans[k])
            cin = chans[k]
        for k in range(levels - 2, -1, -1):  # decoder
            add(cin + chans[k], chans[k])
            add(chans[k], chans[k])
            cin = chans[k]
        self.head_w = torch.nn.Parameter(torch.randn(out_ch, cin, generator=g) * math.sqrt(1.0 / cin))
        self.head_b = torch.nn.Parameter(torch.zeros(out_ch))

    def forward(self, x):
        """x: (B, H, W, IN_CH) BF16, H and W divisible by 2**(levels-1)."""
        i = 0
        skips = []
        for k in range(self.levels):
            x = conv3x3_relu(x, self.ws[i], self.bs[i]); i += 1
            x = conv3x3_relu(x, self.ws[i], self.bs[i]); i += 1
            if k < self.levels - 1:
                skips.append(x)
                x = _pool(x)
        for k in range(self.levels - 2, -1, -1):
            x = conv3x3_up_cat(x, skips[k], self.ws[i], self.bs[i]); i += 1
            x = conv3x3_relu(x, self.ws[i], self.bs[i]); i += 1
        return Conv1x1.apply(x, self.head_w, self.head_b)

    def flops(self, H, W):
        """Multiply-add FLOPs of one forward pass on an H x W input (x2 per MAC)."""
        tot = 0.0
        k = 0
        hh, ww = H, W
        for lv in range(self.levels):
            for _ in range(2):
                cin, cout = self.plan[k]
                tot += 2.0 * 9 * cin * cout * hh * ww
                k += 1
            if lv < self.levels - 1:
                hh, ww = hh // 2, ww // 2
        for lv in range(self.levels - 2, -1, -1):
            hh, ww = hh * 2, ww * 2
            for _ in range(2):
                cin, cout = self.plan[k]
                tot += 2.0 * 9 * cin * cout * hh * ww
                k += 1
        return tot + 2.0 * self.head_w.numel() * H * W


# ---------------------------------------------------------------------------
# features, targets and the guess interface
# ---------------------------------------------------------------------------

def features(H, bed, beta, B):
    """(…, ny, nx) fields -> (B, ny, nx, IN_CH) BF16 normalised inputs."""
    def b3(t):
        t = torch.as_tensor(t)
        return t.unsqueeze(0) if t.dim() == 2 else t
    fs = [b3(t) for t in (H, bed, beta, B)]
    if _plain(*fs) and fs[0].dtype in (torch.float32, torch.float64) and \
            all(t.dtype == fs[0].dtype and t.shape == fs[0].shape for t in fs):
        x = torch.empty(fs[0].shape + (IN_CH,), dtype=torch.bfloat16, device=fs[0].device)
        N.check(_lib().glide_guess_features(N.dtype_code(fs[0].dtype), *(t.data_ptr() for t in fs), x.data_ptr(),
                                            fs[0].numel(), N.stream_handle()), "guess features")
        return x
    H, bed, beta, B = (t.float() for t in fs)
    logb = torch.log(torch.clamp(beta, min=1e-8))
    x = torch.stack([H / 1000.0, bed / 1000.0, (logb + 2.2) / 0.7, B / 35.0], dim=-1)
    pad = torch.zeros(x.shape[:-1] + (IN_CH - x.shape[-1],), device=x.device)
    return torch.cat([x, pad], dim=-1).to(torch.bfloat16).contiguous()


def cell_velocities(u, v):
    """Face velocities -> cell-centred (…, ny, nx, 2) / VEL_SCALE."""
    uc = 0.5 * (u[..., :, 1:] + u[..., :, :-1])
    vc = 0.5 * (v[..., 1:, :] + v[..., :-1, :])
    return torch.stack([uc, vc], dim=-1) / VEL_SCALE


def faces_from_cells(pred):
    """(…, ny, nx, 2) cell velocities (scaled) -> staggered (u, v) in m/a."""
    uc = pred[..., 0] * VEL_SCALE
    vc = pred[..., 1] * VEL_SCALE
    u = torch.cat([uc[..., :, :1], 0.5 * (uc[..., :, 1:] + uc[..., :, :-1]), uc[..., :, -1:]], dim=-1)
    v = torch.cat([vc[..., :1, :], 0.5 * (vc[..., 1:, :] + vc[..., :-1, :]), vc[..., -1:, :]], dim=-2)
    return u, v


class GuessModel:
    """Trained network + the IcePhysics guess interface."""

    def __init__(self, net: UNet):
        self.net = net

    @torch.no_grad()
    def predict(self, H, bed, beta, B):
        x = features(H, bed, beta, B)
        pred = self.net(x).float()
        if _plain(pred) and pred.dim() == 4 and pred.shape[-1] == 2 and pred.data_ptr() % 8 == 0 and \
                pred.shape[0] <= 65535 and pred.shape[1] <= 8 * 65535 - 8:
            nb, ny, nx, _ = pred.shape
            u = torch.empty((nb, ny, nx + 1), dtype=torch.float64, device=pred.device)
            v = torch.empty((nb, ny + 1, nx), dtype=torch.float64, device=pred.device)
            N.check(_lib().glide_guess_faces(pred.data_ptr(), u.data_ptr(), v.data_ptr(), nb, ny, nx, VEL_SCALE,
                                             N.stream_handle()), "guess faces")
        else:
            u, v = (t.double() for t in faces_from_cells(pred))
        if u.shape[0] == 1:
            u, v = u[0], v[0]
        return u, v

    def save(self, path=DEFAULT_WEIGHTS):
        torch.save(self.net.state_dict(), path)


def load_default_model(path=DEFAULT_WEIGHTS, device="cuda"):
    """The trained guess shipped with the package, or None when absent."""
    if not Path(path).exists():
        return None
    net = UNet()
    net.load_state_dict(torch.load(path, map_location="cpu"))
    return GuessModel(net.to(device))
