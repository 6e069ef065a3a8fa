"""The FP64 kernels have a form of their own for Glen's n = 3 (reciprocal cube
root); every operator at n = 3 and at a general exponent against the FP64
oracle, norm-wise relative 1e-10."""
import pytest
import torch

from test_gpu_kernels import TOL, _np, _rel, _state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3.0, 2.5, 4.0])
def test_fp64_operators_by_exponent(n):
    from glide_b200.grid import Grid
    from oracle import ssa
    from oracle.vanka import vanka_adjoint_color, vanka_deltas, vanka_linear_update
    st = _state((33, 47), seed=23)
    for k in ("u", "v"):
        st[k] = st[k] * 0.02
    p = ssa.Params(n=n)
    g = Grid(33, 47, st["dx"], dt=st["dt"], n=n, dtype=torch.float64)
    for k in ("u", "v", "H", "bed", "B", "beta", "mask", "gamma", "f_u", "f_v", "f_H", "d_u", "d_v", "d_H"):
        getattr(g, k).copy_(torch.as_tensor(st[k]))
    U, d, f = ([st[a + b] for b in ("u", "v", "H")] for a in ("", "d_", "f_"))
    geo = (st["bed"], st["B"], st["beta"], st["mask"], st["gamma"], p, st["dx"], st["dt"])
    for a, b in zip((g.lambda_u, g.lambda_v, g.lambda_H), d):
        a.copy_(torch.as_tensor(b))
    g.compute_residual()
    g.compute_jvp()
    g.compute_vjp()
    r, j, l = ssa.residual(*U, *f, *geo), ssa.jvp(*U, *d, *geo), ssa.vjp(*U, *d, *geo)
    pairs = list(zip((g.r_u, g.r_v, g.r_H, g.j_u, g.j_v, g.j_H, g.l_u, g.l_v, g.l_H), (*r, *j, *l)))
    # one linear sweep, one adjoint colour, one nonlinear sweep
    g.vanka_lu(shift=0.0)
    x = torch.zeros_like(g.U)
    g.vanka_linear_sweep(g.r, x, omega=1.0)
    cells = (st["bed"], st["B"], st["beta"], st["gamma"], p, st["dx"], st["dt"])
    zero = 0.0 * st["H"]
    pairs += zip(g._vec_to_fields(x), vanka_linear_update(*U, st["f_H"], *r, zero, *cells, shift=0.0))
    g.r_adj.copy_(g.r)
    g.vanka_smooth_adjoint(0, 1.0)
    pairs += zip((g.lambda_u, g.lambda_v, g.lambda_H), vanka_adjoint_color(*d, st["mask"], r, *U, *cells, 0, 1.0))
    U0 = g.U.clone()
    g.vanka_sweep(1, n_inner=2, omega=1.0, shift=0.0, step=1.0)
    pairs += zip(g._vec_to_fields(g.U - U0), vanka_deltas(*U, *f, *cells, 2, shift=0.0, step=1.0))
    for a, b in pairs:
        assert _rel(_np(a), b) <= TOL["fp64"]
