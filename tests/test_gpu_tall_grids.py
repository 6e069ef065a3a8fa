"""Grids of more rows than a launch has tile rows (65,535 of four rows each):
the last rows get what they get on a grid of their own."""
import pytest
import torch

pytestmark = pytest.mark.gpu

ROWS, TAIL = 262_200, 64


def _pair(dtype):
    from glide_b200.grid import Grid
    gen = torch.Generator(device="cuda").manual_seed(2)

    def rand(*shape):
        return torch.randn(*shape, generator=gen, device="cuda", dtype=torch.float64)

    f = {"u": 0.02 * rand(ROWS, 2), "v": 0.02 * rand(ROWS + 1, 1), "H": 500 + 100 * rand(ROWS, 1).abs(),
         "bed": -100 + 50 * rand(ROWS, 1), "beta": 0.01 + 0.001 * rand(ROWS, 1).abs(), "f_u": 0.01 * rand(ROWS, 2),
         "f_v": 0.01 * rand(ROWS + 1, 1), "f_H": 0.01 * rand(ROWS, 1), "f_adj_u": rand(ROWS, 2),
         "f_adj_v": rand(ROWS + 1, 1), "f_adj_H": rand(ROWS, 1)}
    gs = [Grid(n, 1, 1000.0, 1.0, dtype=dtype) for n in (ROWS, TAIL)]
    for g in gs:
        for k, t in f.items():
            a = getattr(g, k)
            a.copy_(t[t.shape[0] - a.shape[0]:])
        g.B.fill_(100.0), g.gamma.fill_(0.1)
    return gs


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_adjoint_sweep_reaches_the_last_rows(dtype):
    gs = _pair(dtype)
    for g in gs:
        g.vanka_sweep_adjoint(1)
    for k in ("lambda_u", "lambda_v", "lambda_H"):
        a, b = (getattr(g, k)[-20:] for g in gs)
        assert torch.equal(a, b) and float(a.abs().max()) > 0


@pytest.mark.parametrize("sweeps", [1, 2])
def test_tile_sweep_reaches_the_last_rows(sweeps):
    gs = _pair(torch.float32)
    before = gs[0].H[-20:].clone()
    for g in gs:
        g.vanka_sweep(sweeps, n_inner=3)
    for k in ("u", "v", "H"):
        assert torch.equal(*(getattr(g, k)[-20:] for g in gs))
    assert not torch.equal(gs[0].H[-20:], before)
