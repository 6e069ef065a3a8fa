"""The forward sweep at sizes from one tile to many waves of them, on both sides
of its march and chaining rules, against the oracle; a chain of sweeps equals
the same sweeps with a synchronisation after each; FP64 1e-10, FP32 4e-4
(tolerances of test_vanka_sweep)."""
import pytest
import torch

from test_gpu_kernels import TOL, _grid, _np, _params, _rel, _state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("shape", [(33, 20), (64, 128), (65, 128), (130, 131), (200, 130), (301, 330), (1100, 560)])
def test_sweep_by_size(precision, shape):
    from oracle.vanka import vanka_deltas
    st = _state(shape, seed=5)
    for k in ("u", "v"):
        st[k] = st[k] * 0.02
    g = _grid(st, precision)
    g.vanka_sweep(1, n_inner=3, omega=0.5, shift=1.0)
    ref = vanka_deltas(st["u"], st["v"], st["H"], st["f_u"], st["f_v"], st["f_H"], st["bed"], st["B"], st["beta"],
                       st["gamma"], _params(), st["dx"], st["dt"], 3, shift=1.0)
    tol = TOL[precision] * (1 if precision == "fp64" else 20)
    for a, x0, d in zip((g.u, g.v, g.H), (st["u"], st["v"], st["H"]), ref):
        assert _rel(_np(a) - x0, 0.5 * d) <= tol


@pytest.mark.parametrize("shape", [(40, 40), (150, 140), (260, 250)])
def test_chained_sweeps_equal_separate_ones(shape):
    """20 sweeps (and residuals between them) enqueued at once, one by one with
    a synchronisation, and replayed from a graph: the same bits."""
    def run(g, sync):
        for _ in range(20):
            g.vanka_sweep(1, n_inner=2, shift=1.0)
            sync()
            g.compute_residual()
            sync()
            g.f_adj.copy_(g.r)
            g.vanka_sweep_adjoint(1)
            sync()

    st = _state(shape, seed=6)
    for k in ("u", "v"):
        st[k] = st[k] * 0.02
    gs = [_grid(st, "fp32") for _ in range(3)]
    run(gs[0], lambda: None)
    run(gs[1], torch.cuda.synchronize)
    U0, L0 = gs[2].U.clone(), gs[2].Lambda.clone()
    run(gs[2], lambda: None)   # warm-up outside the capture
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        gs[2].U.copy_(U0), gs[2].Lambda.copy_(L0)
        run(gs[2], lambda: None)
    graph.replay()
    torch.cuda.synchronize()
    for g in gs[1:]:
        assert torch.equal(g.U, gs[0].U) and torch.equal(g.r, gs[0].r) and torch.equal(g.Lambda, gs[0].Lambda)
