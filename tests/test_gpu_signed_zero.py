"""Ice at rest: the upwind side of a face follows the sign of its zero velocity
(copysign, glide/cuda/flux.cu:53), in the march, the linear factors and the adjoint
solve as in the oracle; FP64 1e-10."""
import numpy as np
import pytest
import torch

from test_gpu_kernels import _grid, _np, _params, _rel, _state

pytestmark = pytest.mark.gpu

SIGNS = [(0.0, 0.0), (-0.0, 0.0), (0.0, -0.0), (-0.0, -0.0)]


def _rest(shape, zu, zv):
    st = _state(shape, seed=11)
    st["u"], st["v"] = np.full_like(st["u"], zu), np.full_like(st["v"], zv)
    return st


@pytest.mark.parametrize("zu,zv", SIGNS)
def test_march_from_rest(zu, zv):
    from oracle.vanka import vanka_deltas
    st = _rest((37, 61), zu, zv)
    g = _grid(st, "fp64")
    g.vanka_sweep(1, n_inner=3, omega=0.5)
    ref = vanka_deltas(st["u"], st["v"], st["H"], st["f_u"], st["f_v"], st["f_H"], st["bed"], st["B"], st["beta"],
                       st["gamma"], _params(), st["dx"], st["dt"], 3, shift=1.0)
    for a, x0, d in zip((g.u, g.v, g.H), (st["u"], st["v"], st["H"]), ref):
        assert _rel(_np(a) - x0, 0.5 * d) <= 1e-10


@pytest.mark.parametrize("zu,zv", SIGNS)
def test_linear_sweep_at_rest(zu, zv):
    from oracle.vanka import vanka_linear_update
    st = _rest((37, 61), zu, zv)
    g = _grid(st, "fp64")
    rho = torch.as_tensor(np.random.default_rng(9).standard_normal(g.U.numel()), device="cuda")
    d = torch.zeros_like(rho)
    g.vanka_lu(shift=0.0)
    g.vanka_linear_sweep(rho, d, omega=0.5)
    r = [_np(t) for t in g._vec_to_fields(rho)]
    ref = vanka_linear_update(st["u"], st["v"], st["H"], st["f_H"], *r, np.zeros_like(st["H"]), st["bed"], st["B"],
                              st["beta"], st["gamma"], _params(), st["dx"], st["dt"], shift=0.0)
    for a, b in zip(g._vec_to_fields(d), ref):
        assert _rel(_np(a), 0.5 * b) <= 1e-10


@pytest.mark.parametrize("zu,zv", SIGNS)
def test_adjoint_solve_at_rest(zu, zv):
    from oracle.vanka import vanka_adjoint_color
    st = _rest((37, 61), zu, zv)
    g = _grid(st, "fp64")
    r = [st["f_u"], st["f_v"], st["f_H"]]
    for k, t in zip(("r_adj_u", "r_adj_v", "r_adj_H"), r):
        getattr(g, k).copy_(torch.as_tensor(t))
    g.Lambda.zero_()
    g.vanka_smooth_adjoint(0, omega=1.0)
    z = [np.zeros_like(t) for t in r]
    ref = vanka_adjoint_color(*z, st["mask"], r, st["u"], st["v"], st["H"], st["bed"], st["B"], st["beta"], st["gamma"],
                              _params(), st["dx"], st["dt"], 0, 1.0)
    for a, b in zip((g.lambda_u, g.lambda_v, g.lambda_H), ref):
        assert _rel(_np(a), b) <= 1e-10
