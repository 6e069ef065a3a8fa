"""A problem's forward sweeps do not depend on what shares its batch: the form
of the cell kernel is chosen by the problem's own size.  200^2 lies below the
line of 2^16 cells, two or four of them above it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("ny,nx,nb,newton", [(200, 200, 2, 10), (130, 140, 4, 10), (200, 200, 3, 2)])
def test_sweeps_of_a_batch_equal_single_ones(ny, nx, nb, newton, dtype, gated):
    from glide_b200.grid import Grid
    gen = torch.Generator(device="cuda").manual_seed(4)

    def rand(*shape):
        return torch.randn(*shape, generator=gen, device="cuda", dtype=torch.float64)

    fields = {"u": 0.02 * rand(nb, ny, nx + 1), "v": 0.02 * rand(nb, ny + 1, nx), "H": 500 + 100 * rand(nb, ny, nx).abs(),
              "bed": -100 + 50 * rand(nb, ny, nx), "beta": 0.01 + 0.001 * rand(nb, ny, nx).abs(),
              "f_u": 0.01 * rand(nb, ny, nx + 1), "f_v": 0.01 * rand(nb, ny + 1, nx), "f_H": 0.01 * rand(nb, ny, nx)}

    def sweep(pick, n):
        g = Grid(ny, nx, 1000.0, 1.0, dtype=dtype, nb=n)
        for k, t in fields.items():
            getattr(g, k).copy_(pick(t))
        g.B.fill_(100.0), g.gamma.fill_(0.1)
        g.error_mask.zero_()
        g.error_mask[..., : ny // 3, nx // 2:] = 1.0
        (g.vanka_sweep_local if gated else g.vanka_sweep)(3, n_inner=newton)
        return g

    whole = sweep(lambda t: t, nb)
    for b in range(nb):
        one = sweep(lambda t: t[b], 1)
        for k in ("u", "v", "H"):
            assert torch.equal(getattr(whole, k)[b], getattr(one, k)), (b, k)
