"""Local solves that end in infinities or NaN leave their cell and its share of
the faces unchanged: in the march as in the tile (row-pivoted solves, which are
checked against the oracle), and in the one-pass linear sweep."""
import numpy as np
import pytest
import torch

from test_gpu_kernels import _grid, _np, _rel, _state

pytestmark = pytest.mark.gpu

BAD = {"f_u": [((5, 10), np.nan), ((0, 0), np.inf), ((36, 61), -np.inf)], "f_v": [((37, 3), np.inf), ((18, 29), np.nan)],
       "f_H": [((20, 30), np.inf), ((21, 30), np.nan), ((9, 59), -np.inf)]}


def _small(seed):
    st = _state((37, 61), seed=seed)
    for k in ("u", "v"):
        st[k] = st[k] * 0.02
    return st


@pytest.mark.parametrize("gated", [False, True])
def test_march_skips_failed_cells(gated):
    st = _small(3)
    for k, put in BAD.items():
        for at, x in put:
            st[k][at] = x
    a, b = _grid(st, "fp64"), _grid(st, "fp64")
    for g, pivot in ((a, False), (b, True)):
        if gated:
            g.error_mask.zero_()
            g.error_mask[:25, 20:] = 1.0
            g.update_tile_flags()
        g._sweeps(3, 3, 0.5, 1.0, gated, 0.25, pivot)
    assert bool(torch.isfinite(a.U).all())
    for x, y, x0 in zip((a.u, a.v, a.H), (b.u, b.v, b.H), (st["u"], st["v"], st["H"])):
        assert _rel(_np(x) - x0, _np(y) - x0) <= 1e-10


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_linear_sweep_skips_failed_cells(precision):
    st = _small(4)
    g = _grid(st, precision)
    gen = torch.Generator(device="cuda").manual_seed(2)
    rho = torch.randn(g.U.numel(), generator=gen, device="cuda", dtype=g.dtype)
    bad = rho.clone()
    hit = torch.zeros(37, 61, dtype=torch.bool, device="cuda")   # cells that see a bad entry
    for t, (k, put) in zip(g._vec_to_fields(bad), BAD.items()):
        for (i, j), x in put:
            t[i, j] = x
            for a, b in {"f_u": ((i, j - 1), (i, j)), "f_v": ((i - 1, j), (i, j)), "f_H": ((i, j),) * 2}[k]:
                if 0 <= a < 37 and 0 <= b < 61:
                    hit[a, b] = True
    g.vanka_lu(0.0)
    d, e = g._vec(), g._vec()
    g.vanka_linear_sweep(rho, d, 0.5)
    g.vanka_linear_sweep(bad, e, 0.5)
    assert bool(torch.isfinite(e).all())
    (du, dv, dH), (eu, ev, eH) = g._vec_to_fields(d), g._vec_to_fields(e)
    assert bool((eH[hit] == 0).all()) and torch.equal(eH[~hit], dH[~hit])
    fu = torch.nn.functional.pad(hit, (0, 1)) | torch.nn.functional.pad(hit, (1, 0))
    fv = torch.nn.functional.pad(hit, (0, 0, 0, 1)) | torch.nn.functional.pad(hit, (0, 0, 1, 0))
    assert torch.equal(eu[~fu], du[~fu]) and torch.equal(ev[~fv], dv[~fv])
    both = hit[:, 1:] & hit[:, :-1]
    assert bool((eu[:, 1:-1][both] == 0).all())


@pytest.mark.parametrize("P,N", [(1, 8), (1001, 24), (70003, 256), (70003, 40), (4097, 2048)])
def test_bias_gradient_counts_every_pixel(P, N):
    """Whole numbers add up exactly in FP32: any pixel left out or added twice shows
    (P no multiple of what the blocks take at once)."""
    from glide_b200.guess import _relu_grad
    gen = torch.Generator(device="cuda").manual_seed(P)
    gy = torch.randint(-8, 9, (P, N), generator=gen, device="cuda").to(torch.bfloat16)
    y = torch.randint(0, 2, (P, N), generator=gen, device="cuda").to(torch.bfloat16)
    gz, db = _relu_grad(gy, y, True)
    ref = gy.double() * (y > 0)
    assert torch.equal(gz.double(), ref) and torch.equal(db.double(), ref.sum(0))
