"""The marching form of the forward cell kernel (FP64, and FP32 from 2^16 cells
on) at the edges of its 30-column strips and row chunks, whole and gated by
the error mask, against the oracle; FP64 1e-10, FP32 4e-4 (tolerances of
test_vanka_sweep)."""
import pytest
import torch

from test_gpu_kernels import TOL, _grid, _np, _params, _rel, _state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("precision,shape", [("fp64", (1, 2)), ("fp64", (2, 29)), ("fp64", (7, 30)),
                                             ("fp64", (31, 31)), ("fp64", (45, 61)), ("fp64", (301, 453)),
                                             ("fp32", (257, 256)), ("fp32", (2200, 30)), ("fp32", (331, 241))])
def test_march_by_size(precision, shape, gated):
    from oracle.vanka import local_cell_on, vanka_deltas
    st = _state(shape, seed=7)
    for k in ("u", "v"):
        st[k] = st[k] * 0.02
    g = _grid(st, precision)
    on = None
    if gated:
        em = torch.zeros(shape)
        em[: max(1, shape[0] // 3), shape[1] // 2:] = 1.0
        g.error_mask.copy_(em.to(g.error_mask))
        on = local_cell_on(em.numpy())
        g.vanka_sweep_local(1, n_inner=3, omega=0.5)
    else:
        g.vanka_sweep(1, n_inner=3, omega=0.5)
    ref = vanka_deltas(st["u"], st["v"], st["H"], st["f_u"], st["f_v"], st["f_H"], st["bed"], st["B"], st["beta"],
                       st["gamma"], _params(), st["dx"], st["dt"], 3, shift=1.0, cell_on=on)
    tol = TOL[precision] * (1 if precision == "fp64" else 20)
    for a, x0, d in zip((g.u, g.v, g.H), (st["u"], st["v"], st["H"]), ref):
        assert _rel(_np(a) - x0, 0.5 * d) <= tol
