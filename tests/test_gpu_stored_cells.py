"""Stored local systems: the linear sweep in one pass and the adjoint sweeps
from kept factors, against the FP64 oracle and the per-colour entry point, at
widths around the strips (30 and 31 columns), one row or column, a batch, and
chunks of one and of several rows.

Tolerances (norm-wise relative): FP64 1e-10 and FP32 2e-5 per application as in
test_gpu_kernels; the FP32 adjoint sweeps apply 2 colours x 2 sweeps (4x)."""
import ctypes as C

import numpy as np
import pytest
import torch

from test_gpu_kernels import TOL, _grid, _np, _params, _rel, _state

pytestmark = pytest.mark.gpu

SHAPES = [(1, 2), (1, 40), (37, 1), (5, 30), (8, 31), (9, 32), (40, 61), (70, 93), (200, 190)]


def _small(shape, seed):
    st = _state(shape, seed=seed)
    for k in ("u", "v"):
        st[k] = st[k] * 0.02
    return st


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("shape", SHAPES)
def test_adjoint_sweeps_from_factors(precision, shape):
    """Sweeps from kept factors = the same sweeps colour by colour through the
    entry points that form the systems each time (checked against the oracle in
    test_gpu_kernels)."""
    st = _small(shape, 13)
    a, b = (_grid(st, precision, gl_derivatives=True) for _ in range(2))
    g = torch.Generator().manual_seed(5)
    for n in ("f_adj", "Lambda"):
        t = torch.randn(a.U.numel(), generator=g, dtype=torch.float64)
        getattr(a, n).copy_(t), getattr(b, n).copy_(t)
    a.vanka_sweep_adjoint(2, omega=0.7, exact_boundary=True)
    for _ in range(2):
        for color in (0, 1):
            b.compute_adjoint_residual(True)
            b.vanka_smooth_adjoint(color, 0.7)
    for x, y in zip((a.lambda_u, a.lambda_v, a.lambda_H), (b.lambda_u, b.lambda_v, b.lambda_H)):
        assert _rel(_np(x), _np(y)) <= 4 * TOL[precision]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("shape", SHAPES)
def test_linear_sweep_vs_oracle(precision, shape):
    """The one-pass linear sweep against the oracle (tolerances of
    test_vanka_linear_sweep_vs_oracle: 1e-10 and 2e-4)."""
    from oracle.vanka import vanka_linear_update
    st = _small(shape, 17)
    g = _grid(st, precision)
    rng = np.random.default_rng(9)
    rho = torch.as_tensor(rng.standard_normal(g.U.numel()), dtype=g.dtype, device="cuda")
    d = torch.as_tensor(rng.standard_normal(g.U.numel()) * 0.1, dtype=g.dtype, device="cuda")
    d0 = d.clone()
    g.vanka_lu(shift=0.0)
    g.vanka_linear_sweep(rho, d, omega=0.5)
    r, x0 = ([_np(t) for t in g._vec_to_fields(v)] for v in (rho, d0))
    ref = vanka_linear_update(st["u"], st["v"], st["H"], st["f_H"], *r, x0[2], st["bed"], st["B"], st["beta"],
                              st["gamma"], _params(), st["dx"], st["dt"], shift=0.0)
    for a, b, z in zip(g._vec_to_fields(d), ref, x0):
        assert _rel(_np(a) - z, 0.5 * b) <= (1e-10 if precision == "fp64" else 2e-4)


def test_linear_and_adjoint_batch_equal_single():
    from glide_b200.grid import Grid
    sts = [_small((33, 47), s) for s in (20, 21, 22)]
    g = Grid(33, 47, sts[0]["dx"], dt=10.0, dtype=torch.float32, nb=3)
    names = ("u", "v", "H", "bed", "B", "beta", "mask", "gamma", "f_u", "f_v", "f_H")
    for k in names:
        getattr(g, k).copy_(torch.as_tensor(np.stack([s[k] for s in sts])))

    def go(x):
        x.compute_residual()
        x.vanka_lu(0.0)
        x.d_U.zero_()
        x.vanka_linear_sweep(x.r, x.d_U, 0.5)
        x.f_adj.copy_(x.r)
        x.Lambda.zero_()
        x.vanka_sweep_adjoint(1)

    go(g)
    for b, st in enumerate(sts):
        s = _grid(st, "fp32")
        go(s)
        for n in ("d_u", "d_v", "d_H", "lambda_u", "lambda_v", "lambda_H"):
            assert torch.equal(getattr(g, n)[b], getattr(s, n)), n
