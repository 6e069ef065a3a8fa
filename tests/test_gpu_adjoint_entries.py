"""The adjoint V-cycle is the same through the physics object and through the
exported function: both keep the smoother's systems, level by level."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_exported_cycle_equals_the_method(precision):
    from glide_b200 import IcePhysics, adjoint_vcycle
    from glide_b200.solver import hierarchy
    from glide_b200.synthetic import dome_case

    def solved():
        c = dome_case(3, n=64, dx=10000.0)
        ph = IcePhysics(64, 64, c.dx, n_levels=3, precision=precision)
        ph.set_geometry(c.bed, c.thickness)
        ph.set_parameters(B=c.B, beta=c.beta, smb=c.smb)
        ph.forward(c.dt, n_vcycles=1, update_geometry=False)
        return ph

    a, b = solved(), solved()
    gen = torch.Generator(device="cuda").manual_seed(1)
    d = [torch.randn(t.shape, generator=gen, device="cuda", dtype=t.dtype) for t in (a.grid.u, a.grid.v, a.grid.H)]
    a.adjoint(*d, n_vcycles=2)
    g = b.grid
    g.f_adj_u.copy_(-d[0]), g.f_adj_v.copy_(-d[1]), g.f_adj_H.copy_(-d[2])
    g.Lambda.zero_()
    for _ in range(2):
        adjoint_vcycle(g, b.settings, b.thklim)
    assert all(x._adj_factors is not None for x in hierarchy(g))
    assert torch.equal(a.grid.Lambda, g.Lambda) and float(g.Lambda.abs().max()) > 0
