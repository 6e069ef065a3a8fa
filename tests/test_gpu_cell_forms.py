"""Both forms of the forward cell kernel on both sides of the rule that chooses
one (type, size, Newton steps, gating), against the oracle: FP64 1e-10, FP32
4e-4 (tolerances of test_vanka_sweep).  Beside test_gpu_cell_march: the march
with the step counts that take it, and the tile in FP64 (gated, from 512^2 on)."""
import pytest
import torch

from test_gpu_kernels import TOL, _grid, _np, _params, _rel, _state

pytestmark = pytest.mark.gpu


def _small(shape, seed):
    st = _state(shape, seed=seed)
    for k in ("u", "v"):
        st[k] = st[k] * 0.02
    return st


def _gate(g, shape):
    g.error_mask.zero_()
    g.error_mask[: max(1, shape[0] // 3), shape[1] // 2:] = 1.0


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("precision,shape,newton", [
    ("fp32", (257, 256), 8), ("fp32", (2200, 30), 8), ("fp32", (331, 241), 8), ("fp32", (640, 621), 2),
    ("fp32", (731, 725), 2), ("fp64", (1, 2), 2), ("fp64", (33, 31), 2), ("fp64", (131, 65), 2), ("fp64", (256, 257), 2),
    ("fp64", (513, 514), 3), ("fp64", (513, 514), 8), ("fp64", (700, 702), 2), ("fp64", (730, 731), 2)])
def test_form_by_size(precision, shape, newton, gated):
    from oracle.vanka import local_cell_on, vanka_deltas
    st = _small(shape, 9)
    g = _grid(st, precision)
    on = None
    if gated:
        _gate(g, shape)
        on = local_cell_on(g.error_mask.cpu().numpy())
    (g.vanka_sweep_local if gated else g.vanka_sweep)(1, n_inner=newton, omega=0.5)
    ref = vanka_deltas(st["u"], st["v"], st["H"], st["f_u"], st["f_v"], st["f_H"], st["bed"], st["B"], st["beta"],
                       st["gamma"], _params(), st["dx"], st["dt"], newton, shift=1.0, cell_on=on)
    tol = TOL[precision] * (1 if precision == "fp64" else 20)
    for a, x0, d in zip((g.u, g.v, g.H), (st["u"], st["v"], st["H"]), ref):
        assert _rel(_np(a) - x0, 0.5 * d) <= tol
