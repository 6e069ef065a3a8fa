"""The arrow-form local solves over FP32's range: with B = 0 every face is its
drag alone, so FP32 has to agree with FP64 at any size of the drag that both
hold (relative 1e-5: a few FP32 roundings)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _grid(ny, nx, dtype, beta):
    from glide_b200.grid import Grid
    gen = torch.Generator(device="cuda").manual_seed(1)

    def rand(*shape):
        return torch.randn(*shape, generator=gen, device="cuda")

    g = Grid(ny, nx, 1000.0, 1.0, dtype=dtype)
    for k, t in (("u", rand(ny, nx + 1)), ("v", rand(ny + 1, nx)), ("H", 500 + 10 * rand(ny, nx)),
                 ("beta", beta * (1 + 0.1 * rand(ny, nx).abs())), ("lambda_u", 0 * rand(ny, nx + 1)),
                 ("f_adj_u", rand(ny, nx + 1)), ("f_adj_v", rand(ny + 1, nx))):
        getattr(g, k).copy_(t)
    g.bed.fill_(1000.0), g.B.zero_(), g.gamma.fill_(0.1), g.f_H.copy_(g.H)
    return g


def _near(a, b):
    return float((a.double() - b).norm() / b.norm()) <= 1e-5


@pytest.mark.parametrize("beta", [1e-3, 1.0, 1e10, 2.4e19, 1e25, 1e30])
def test_adjoint_solve_at_any_drag(beta):
    out = []
    for dtype in (torch.float32, torch.float64):
        g = _grid(9, 37, dtype, beta)
        g.r_adj_u.copy_(g.f_adj_u), g.r_adj_v.copy_(g.f_adj_v), g.r_adj_H.zero_()
        g.vanka_smooth_adjoint(0, 1.0)
        out.append((g.lambda_u.double() * beta, g.lambda_v.double() * beta))
    assert all(_near(a, b) for a, b in zip(*out))


@pytest.mark.parametrize("beta", [1e-3, 1.0, 1e10, 2.4e19, 1e25, 1e30])
def test_linear_sweep_at_any_drag(beta):
    out = []
    for dtype in (torch.float32, torch.float64):
        g = _grid(9, 37, dtype, beta)
        g.vanka_lu(0.0)
        rho, d = g._vec(), g._vec()
        ru, rv, _ = g._vec_to_fields(rho)
        ru.copy_(g.f_adj_u), rv.copy_(g.f_adj_v)
        g.vanka_linear_sweep(rho, d, 0.5)
        out.append([t.double() * beta for t in g._vec_to_fields(d)[:2]])
    assert all(_near(a, b) for a, b in zip(*out))


@pytest.mark.parametrize("beta", [1e10, 2.4e19, 1e25, 1e30])
def test_march_at_any_drag(beta):
    """Undamped steps without shift: a drag this large halves the velocities with
    every sweep, to 2^-30 of what they were (and rounding)."""
    g = _grid(257, 260, torch.float32, beta)
    u0 = float(g.u.abs().max())
    for _ in range(30):
        g.vanka_sweep(1, n_inner=8, omega=0.5, shift=0.0, step=1.0)
    assert max(float(g.u[:, 1:-1].abs().max()), float(g.v[1:-1].abs().max())) <= 2.0 ** -20 * u0
