"""Sweeps that pass the state on inside the cell kernel (one kernel per sweep)
give the bits of separate calls, each a cell kernel and an update: whole and
gated, at edges of the tiles, odd and even sweep counts, and a batch in
which one scenario has no active cell."""
import pytest
import torch

from test_gpu_kernels import _grid, _state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("n", [2, 3, 10])
@pytest.mark.parametrize("shape", [(1, 2), (3, 33), (33, 20), (64, 65), (65, 128), (130, 131), (250, 260)])
def test_fused_sweeps_equal_single_ones(shape, n, gated):
    st = _state(shape, seed=8)
    for k in ("u", "v"):
        st[k] = st[k] * 0.02
    a, b = _grid(st, "fp32"), _grid(st, "fp32")
    for g in (a, b):
        g.error_mask.zero_()
        g.error_mask[: max(1, shape[0] // 3), shape[1] // 2:] = 1.0
    sweep = "vanka_sweep_local" if gated else "vanka_sweep"
    getattr(a, sweep)(n, n_inner=3)
    for _ in range(n):
        getattr(b, sweep)(1, n_inner=3)
    assert torch.equal(a.U, b.U)


def test_fused_sweeps_of_a_batch():
    from glide_b200.grid import Grid
    gs = [Grid(45, 70, 1000.0, 1.0, dtype=torch.float32, nb=3) for _ in range(2)]
    gen = torch.Generator(device="cuda").manual_seed(1)
    U = torch.randn(gs[0].U.shape, generator=gen, device="cuda") * 0.02
    f = torch.randn(gs[0].U.shape, generator=gen, device="cuda") * 0.01
    for g in gs:
        g.U.copy_(U), g.f.copy_(f)
        g.H.copy_(500 + 100 * g.H)
        g.bed.fill_(-100.0), g.B.fill_(100.0), g.beta.fill_(0.01), g.gamma.fill_(0.1)
        g.error_mask.zero_()
        g.error_mask[0, 5:20, 30:] = 1.0
        g.error_mask[2, 40:, :9] = 1.0
    gs[0].vanka_sweep_local(5, n_inner=3)
    for _ in range(5):
        gs[1].vanka_sweep_local(1, n_inner=3)
    assert bool(torch.isfinite(gs[0].U).all())
    assert torch.equal(gs[0].U, gs[1].U) and not torch.equal(gs[0].U, U)
    assert torch.equal(gs[0].H[1], 500 + 100 * gs[0]._vec_to_fields(U)[2][1])
