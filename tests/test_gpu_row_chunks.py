"""Marching kernels at sizes whose chunks have 1, 2, 5, 8 and more rows (the
rule follows the number of warps), with a ragged last chunk and strip, against
the FP64 oracle; tolerances of test_gpu_kernels (norm-wise relative)."""
import pytest

from test_gpu_kernels import TOL, _grid, _np, _params, _rel, _state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("shape", [(61, 31), (157, 149), (291, 271), (433, 331), (1210, 1203)])
def test_marches_by_chunk_size(precision, shape):
    import torch
    from oracle import ssa
    st = _state(shape, seed=11)
    g = _grid(st, precision)
    p = _params()
    geo = (st["bed"], st["B"], st["beta"], st["mask"], st["gamma"], p, st["dx"], st["dt"])
    U, d = (st["u"], st["v"], st["H"]), (st["d_u"], st["d_v"], st["d_H"])
    g.compute_residual()
    g.compute_jvp()
    for a, b in zip((g.lambda_u, g.lambda_v, g.lambda_H), d):
        a.copy_(torch.as_tensor(b))
    g.compute_vjp()
    got = (g.r_u, g.r_v, g.r_H, g.j_u, g.j_v, g.j_H, g.l_u, g.l_v, g.l_H)
    ref = (*ssa.residual(*U, st["f_u"], st["f_v"], st["f_H"], *geo), *ssa.jvp(*U, *d, *geo), *ssa.vjp(*U, *d, *geo))
    for a, b in zip(got, ref):
        assert _rel(_np(a), b) <= TOL[precision]
