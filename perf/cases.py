"""Timed cases of the SSA forward/adjoint path and of its learned guess.

Each case is one call (or one short sequence of calls) that a program makes
through the public classes: ``Grid`` operators and smoothers on one level,
``IcePhysics.forward`` / ``adjoint`` with the default settings, the learned
guess and one training layer of it.  ``exact`` restates the Grid operators and
the network in plain FP64 torch.
"""
import math

import torch
import torch.nn.functional as F

RR = 0.917            # rho_ice / rho_water
GLEN, EPS, DRAG, CALV, SIG = 3.0, 1e-5, 1e-3, 1.0, 0.1   # IcePhysics' defaults
THK, DT = 0.1, 10.0
VEL = 100.0           # m/a per unit of the network's output
DTYPES = {"fp32": torch.float32, "fp64": torch.float64}


def listed():
    return [
        # smallest call: residual and its norms on the 64^2 dome grid (a tolerance check)
        {"name": "residual_64_fp64", "kind": "residual", "ny": 64, "nx": 64, "dx": 5000.0, "dtype": "fp64"},
        # largest grid: the residual of the 4096^2 marine sheet in FP32
        {"name": "residual_4096_fp32", "kind": "residual", "ny": 4096, "nx": 4096, "dx": 1000.0, "dtype": "fp32"},
        # the adjoint's FP64 gradient accumulation at 1024^2: masked VJP and basal-friction gradient
        {"name": "gradient_1024_fp64", "kind": "gradient", "ny": 1024, "nx": 1024, "dx": 1000.0, "dtype": "fp64"},
        # pre-smoothing of a V-cycle's finest level at 1024^2 with the default settings
        {"name": "smooth_1024_fp32", "kind": "smooth", "ny": 1024, "nx": 1024, "dx": 1000.0, "dtype": "fp32",
         "sweeps": 10, "newton": 10, "step": 0.25, "shift": 1.0},
        # coarsest-level solve of the 1024^2, 6-level hierarchy: 200 sweeps on 32^2
        {"name": "smooth_32_fp32", "kind": "smooth", "ny": 32, "nx": 32, "dx": 32000.0, "dtype": "fp32",
         "sweeps": 200, "newton": 10, "step": 0.25, "shift": 1.0},
        # one finishing block in FP64 on a regional grid of ragged size: full local Newton steps
        {"name": "smooth_ragged_fp64", "kind": "smooth", "ny": 301, "nx": 453, "dx": 2000.0, "dtype": "fp64",
         "sweeps": 20, "newton": 2, "step": 1.0, "shift": 0.0},
        # linearised FP32 finishing block (factor once, 20 linear sweeps on r + J d), ragged size
        {"name": "linear_ragged_fp32", "kind": "linear", "ny": 1021, "nx": 1403, "dx": 1000.0, "dtype": "fp32",
         "sweeps": 20},
        # adjoint smoothing of a 512^2 level: 10 two-colour sweeps
        {"name": "adjoint_smooth_512_fp32", "kind": "adjoint_smooth", "ny": 512, "nx": 512, "dx": 1500.0,
         "dtype": "fp32", "sweeps": 10},
        # one implicit step with the defaults (FP32, 3 V-cycles): 512^2, 5 levels, the quick-start size
        {"name": "forward_512_fp32", "kind": "forward", "ny": 512, "nx": 512, "dx": 1500.0, "dtype": "fp32",
         "levels": 5, "cycles": 3},
        # the gradient of one step in FP64 (2 adjoint V-cycles), 256^2, 4 levels
        {"name": "adjoint_256_fp64", "kind": "adjoint", "ny": 256, "nx": 256, "dx": 1500.0, "dtype": "fp64",
         "levels": 4, "cycles": 2},
        # learned initial guess of a 1024^2 geometry
        {"name": "guess_1024", "kind": "guess", "ny": 1024, "nx": 1024, "dx": 1000.0},
        # forward and backward of one 3x3 layer on a training batch of eight 256^2 patches
        {"name": "conv_train_256", "kind": "conv_train", "batch": 8, "ny": 256, "nx": 256, "cin": 32, "cout": 32},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["residual", "gradient", "smooth", "smooth", "linear", "adjoint_smooth", "forward", "adjoint",
                       "guess", "conv_train"])
    c = {"kind": kind}
    if kind == "conv_train":
        lv = rng.randrange(4)
        c.update(batch=rng.randint(1, 8), ny=_size(rng, 32, 256) >> lv, nx=_size(rng, 32, 256) >> lv)
        c["cin"] = rng.choice([8, 32, 64, 96, 128, 192])
        c["cout"] = 32 << lv
        return c
    if kind == "guess":
        return dict(c, ny=8 * _size(rng, 8, 128), nx=8 * _size(rng, 8, 128), dx=1000.0)
    if kind in ("forward", "adjoint"):
        lv = rng.randint(2, 5)
        q = 1 << (lv - 1)
        top = 512 if kind == "forward" else 256
        c.update(ny=q * max(3, _size(rng, 48, top) // q), nx=q * max(3, _size(rng, 48, top) // q), levels=lv,
                 cycles=rng.randint(1, 2))
        c.update(dx=float(rng.choice([1000, 1500, 2000, 5000])),
                 dtype="fp32" if kind == "forward" else rng.choice(["fp32", "fp64"]))
        return c
    top = {"residual": 4096, "gradient": 1448, "smooth": 1024, "linear": 1400, "adjoint_smooth": 512}[kind]
    c.update(ny=_size(rng, 17, top), nx=_size(rng, 17, top), dx=float(rng.choice([1000, 1500, 2000, 5000])),
             dtype=rng.choice(["fp32", "fp64"]))
    if kind == "smooth":
        c.update(rng.choice([dict(newton=10, step=0.25, shift=1.0), dict(newton=2, step=1.0, shift=0.0)]))
        c["sweeps"] = rng.randint(4, 10) if c["dtype"] == "fp32" else rng.randint(1, 4)
    elif kind == "linear":
        c.update(dtype="fp32", sweeps=rng.randint(4, 20))
    elif kind == "adjoint_smooth":
        c["sweeps"] = rng.randint(2, 10) if c["dtype"] == "fp32" else rng.randint(1, 4)
    return c


# ------------------------------------------------------------------ inputs

def _field(gen, ny, nx, cells):
    """Smooth random field of unit variance, correlation length in cells."""
    w = torch.randn(ny, nx, generator=gen, device="cuda", dtype=torch.float64)
    ky = torch.fft.fftfreq(ny, device="cuda", dtype=torch.float64)[:, None]
    kx = torch.fft.rfftfreq(nx, device="cuda", dtype=torch.float64)[None, :]
    f = torch.fft.irfft2(torch.fft.rfft2(w) * torch.exp(-(math.pi * cells) ** 2 * (ky ** 2 + kx ** 2)), s=(ny, nx))
    return f / f.std()


def _scene(case, seed):
    """A seeded ice dome, grounded in the middle and afloat in the lows of its
    margin, with a radial flow of a few 100 m/a, in FP64."""
    ny, nx, dx = case["ny"], case["nx"], case["dx"]
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    y = torch.arange(ny, device="cuda", dtype=torch.float64)[:, None]
    x = torch.arange(nx, device="cuda", dtype=torch.float64)[None, :]
    off = 0.1 * (torch.rand(2, generator=gen, device="cuda", dtype=torch.float64) - 0.5)
    top = 1500.0 + 1500.0 * torch.rand((), generator=gen, device="cuda", dtype=torch.float64)

    def rad(ys, xs):   # offsets from the centre, in dome radii
        return (ys / ny - 0.5 - off[0]) / 0.38, (xs / nx - 0.5 - off[1]) / 0.38

    Y, X = rad(y + 0.5, x + 0.5)
    r2 = Y ** 2 + X ** 2
    scale = max(2.0, min(ny, nx) / 12.0)
    s = {"bed": -80.0 * r2 + 150.0 * _field(gen, ny, nx, scale) + 20.0 * _field(gen, ny, nx, 2.0)}
    s["H"] = top * torch.clamp(1.0 - r2, min=0.0) + THK
    s["beta"] = 0.1112 * torch.exp(0.5 * _field(gen, ny, nx, max(2.0, 20e3 / dx)))
    s["B"] = torch.full((ny, nx), 35.18, device="cuda", dtype=torch.float64)
    s["smb"] = 0.5 - 1e-3 * (s["H"] + torch.maximum(s["bed"], -RR * s["H"]) - 1000.0)
    for name, sh, (Ys, Xs) in (("u", (ny, nx + 1), rad(y + 0.5, x.new_tensor(range(nx + 1))[None, :])),
                               ("v", (ny + 1, nx), rad(y.new_tensor(range(ny + 1))[:, None], x + 0.5))):
        flow = (Xs if name == "u" else -Ys) * torch.exp(-(Ys ** 2 + Xs ** 2) ** 2)
        s[name] = 150.0 * flow.expand(sh) + 10.0 * _field(gen, *sh, scale) + 0.2 * _field(gen, *sh, 1.0)
        s["l" + name] = _field(gen, *sh, 3.0) * 1e-2
        s["f" + name] = _field(gen, *sh, 4.0) * 1e-3
    s["lH"] = _field(gen, ny, nx, 3.0) * 1e-2
    s["fH"] = s["H"] / DT + s["smb"]
    return s


def _grid(case, s):
    from glide_b200.grid import Grid
    g = Grid(case["ny"], case["nx"], case["dx"], dt=DT, dtype=DTYPES[case["dtype"]])
    for k in ("u", "v", "H", "bed", "beta", "B", "smb"):
        getattr(g, k).copy_(s[k])
    g.f_u.copy_(s["fu"]), g.f_v.copy_(s["fv"]), g.f_H.copy_(s["fH"])
    g.gamma.fill_(THK)
    return g


def _conv_inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    b, ny, nx, ci, co = (case[k] for k in ("batch", "ny", "nx", "cin", "cout"))
    x = torch.relu(torch.randn(b, ny, nx, ci, generator=gen, device="cuda")).to(torch.bfloat16)
    W = torch.randn(co, 9 * ci, generator=gen, device="cuda") * math.sqrt(2.0 / (9 * ci))
    bias = 0.1 * torch.randn(co, generator=gen, device="cuda")
    gy = (torch.randn(b, ny, nx, co, generator=gen, device="cuda") / (b * ny * nx)).to(torch.bfloat16)
    return x, W, bias, gy


def prepare(case, seed):
    kind = case["kind"]
    if kind == "conv_train":
        x, W, bias, gy = _conv_inputs(case, seed)
        return {"case": case, "x": x.requires_grad_(), "W": W.requires_grad_(), "b": bias.requires_grad_(), "gy": gy}
    s = _scene(case, seed)
    if kind == "guess":
        from glide_b200.guess import load_default_model
        return {"case": case, "model": load_default_model(), "in": [s[k] for k in ("H", "bed", "beta", "B")]}
    if kind in ("forward", "adjoint"):
        from glide_b200 import IcePhysics
        ph = IcePhysics(case["ny"], case["nx"], case["dx"], n_levels=case["levels"], precision=case["dtype"])
        ph.set_geometry(s["bed"], s["H"])
        ph.set_parameters(B=s["B"], beta=s["beta"], smb=s["smb"])
        st = {"case": case, "ph": ph}
        if kind == "adjoint":   # a solved step leaves its state on every level
            from glide_b200.kernels import restrict_cell_centered, restrict_hfacet, restrict_vfacet
            ph._set_dt(DT)
            ph.grid.u.copy_(s["u"]), ph.grid.v.copy_(s["v"])
            for f, c in zip(ph.grids[:-1], ph.grids[1:]):
                restrict_vfacet(f.u, None, c.u), restrict_hfacet(f.v, None, c.v), restrict_cell_centered(f.H, None, c.H)
            st["dL"] = [s[k].to(ph.dtype) for k in ("lu", "lv", "lH")]
        return st
    g = _grid(case, s)
    st = {"case": case, "g": g, "U0": g.U.clone()}
    if kind == "gradient":
        g.lambda_u.copy_(s["lu"]), g.lambda_v.copy_(s["lv"]), g.lambda_H.copy_(s["lH"])
    if kind == "adjoint_smooth":
        g.f_adj_u.copy_(s["lu"]), g.f_adj_v.copy_(s["lv"]), g.f_adj_H.copy_(s["lH"])
    return st


# ------------------------------------------------------------------ one pass

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "conv_train":
        from glide_b200.guess import conv3x3_relu
        y = conv3x3_relu(state["x"], state["W"], state["b"])
        return [y.detach(), *torch.autograd.grad(y, (state["x"], state["W"], state["b"]), state["gy"])]
    if kind == "guess":
        return list(state["model"].predict(*state["in"]))
    if kind == "forward":
        ph = state["ph"]
        ph.reset_solution()
        return list(ph.forward(DT, n_vcycles=case["cycles"], update_geometry=False))
    if kind == "adjoint":
        return state["ph"].adjoint(*state["dL"], n_vcycles=case["cycles"])
    g = state["g"]
    if kind == "residual":
        g.compute_residual()
        return [g.r_u, g.r_v, g.r_H, g.residual_norms()]
    if kind == "gradient":
        g.compute_mask()
        g.compute_vjp(exact_boundary=True)
        return [g.l_u, g.l_v, g.l_H, g.compute_grad_beta(exact_boundary=True)]
    if kind == "smooth":   # a sweep works in place: every pass starts from the same state
        g.U.copy_(state["U0"])
        g.vanka_sweep(case["sweeps"], n_inner=case["newton"], shift=case["shift"], step=case["step"])
        return [g.u, g.v, g.H]
    if kind == "linear":
        g.compute_residual()
        g.vanka_lu(0.0)
        g.d_U.zero_()
        rho = g.r
        for k in range(case["sweeps"]):
            if k:
                g.jvp_add(g.r, g.z)
                rho = g.z
            g.vanka_linear_sweep(rho, g.d_U, 0.5)
        return [g.d_u, g.d_v, g.d_H]
    g.compute_mask()
    g.Lambda.zero_()
    g.vanka_sweep_adjoint(case["sweeps"], omega=1.0)
    return [g.lambda_u, g.lambda_v, g.lambda_H]


# ------------------------------------------------------------------ least work

def _net_work(ny, nx):
    """(flops, activations written) of the 4-level, 32-channel U-Net."""
    ch = [32, 64, 128, 256]
    convs = [(lv, ci, ch[lv]) for lv in range(4) for ci in ((8 if lv == 0 else ch[lv - 1]), ch[lv])]
    convs += [(lv, ci, ch[lv]) for lv in (2, 1, 0) for ci in (ch[lv + 1] + ch[lv], ch[lv])]
    return sum(18.0 * ci * co * (ny >> lv) * (nx >> lv) for lv, ci, co in convs) + 2 * 64.0 * ny * nx


def work(case):
    kind, n = case["kind"], case["ny"] * case["nx"]
    w = 8 if case.get("dtype") == "fp64" else 4
    if kind == "conv_train":   # x, gy and y read or written once in BF16, three products
        p, ci, co = n * case["batch"], case["cin"], case["cout"]
        return {"bytes": 2.0 * p * (2 * ci + 2 * co), "flops": 3 * 18.0 * ci * co * p}
    if kind == "guess":        # 4 fields in, 2 out; the activations could stay on the chip
        return {"bytes": 48.0 * n, "flops": _net_work(case["ny"], case["nx"])}
    if kind == "residual":
        return {"bytes": 14.0 * w * n, "flops": 330.0 * n}
    if kind == "gradient":
        return {"bytes": 14.0 * w * n, "flops": 800.0 * n}
    if kind == "smooth":       # 3 state arrays in and out, 7 fields in; viscosity and Newton steps per sweep
        return {"bytes": 13.0 * w * n, "flops": (160.0 + 450.0 * case["newton"]) * case["sweeps"] * n}
    if kind == "linear":       # residual, factors, then one JVP and one 5x5 substitution per sweep
        return {"bytes": 13.0 * w * n, "flops": (1000.0 + 650.0 * case["sweeps"]) * n}
    if kind == "adjoint_smooth":
        return {"bytes": 16.0 * w * n, "flops": (600.0 + 1700.0 * case["sweeps"]) * n}
    tot = sum(0.25 ** k for k in range(case["levels"]))
    if kind == "forward":      # 20 full sweeps of 10 Newton steps per level and cycle, 200 on the coarsest
        q = n * 0.25 ** (case["levels"] - 1)
        return {"bytes": 13.0 * w * n, "flops": case["cycles"] * 4660.0 * (20.0 * tot * n + 180.0 * q)}
    return {"bytes": 14.0 * w * n, "flops": case["cycles"] * 20 * 1700.0 * tot * n}


# ------------------------------------------------------------------ FP64 restatement

def _cl(a, di, dj):
    """a[i + di, j + dj] with indices clamped to the field."""
    i = torch.arange(a.shape[-2], device=a.device).add(di).clamp(0, a.shape[-2] - 1)
    j = torch.arange(a.shape[-1], device=a.device).add(dj).clamp(0, a.shape[-1] - 1)
    return a[..., i, :][..., j]


def _sig(z):
    return torch.sigmoid(torch.clamp(SIG * z, -20.0, 20.0))


def _surf(bed, H):
    return H + torch.maximum(bed, -RR * H)


def _zpad(a, l, r, t, b):
    return F.pad(a, (l, r, t, b))


def _shear(u, v, dx):
    """Shear rate at every vertex, zero on the boundary."""
    e = 0.5 * ((u[:-1, 1:-1] - u[1:, 1:-1]) + (v[1:-1, 1:] - v[1:-1, :-1])) / dx
    return _zpad(e, 1, 1, 1, 1)


def _eta(s, u, v, dx):
    ux, vy = (u[:, 1:] - u[:, :-1]) / dx, (v[:-1] - v[1:]) / dx
    e = _shear(u, v, dx) ** 2
    e2 = 0.25 * (e[:-1, :-1] + e[:-1, 1:] + e[1:, :-1] + e[1:, 1:])
    return 0.5 * s["B"] * (ux ** 2 + vy ** 2 + ux * vy + e2 + EPS) ** ((1.0 - GLEN) / (2.0 * GLEN))


def _operator(s, dx, u, v, H, beta=None):
    """F(U): momentum on the faces, mass on the cells (the grounded fraction
    carries no derivative, as with gl_derivatives=False)."""
    beta = s["beta"] if beta is None else beta
    bed, d = s["bed"], 1.0 / dx
    g = _sig(bed + RR * H).detach()
    eH = _eta(s, u, v, dx) * H
    ux, vy = (u[:, 1:] - u[:, :-1]) * d, (v[:-1] - v[1:]) * d
    sxx, syy = 2 * eH * (2 * ux + vy), 2 * eH * (ux + 2 * vy)
    ev = _zpad(0.25 * (eH[:-1, :-1] + eH[:-1, 1:] + eH[1:, :-1] + eH[1:, 1:]), 1, 1, 1, 1)
    sxy = 2 * ev * _shear(u, v, dx)
    be = g * beta + (1 - g) * DRAG
    S = _surf(bed, H)
    px, py = torch.cat([be[:, :1], be, be[:, -1:]], 1), torch.cat([be[:1], be, be[-1:]], 0)
    Ru = (_zpad(sxx, 0, 1, 0, 0) - _zpad(sxx, 1, 0, 0, 0) + sxy[:-1] - sxy[1:]) * d - 0.5 * (px[:, 1:] + px[:, :-1]) * u
    Ru = Ru - _zpad(0.5 * (H[:, 1:] + H[:, :-1]) * (S[:, 1:] - S[:, :-1]) * d, 1, 1, 0, 0)
    Rv = (_zpad(syy, 0, 0, 1, 0) - _zpad(syy, 0, 0, 0, 1) + sxy[:, 1:] - sxy[:, :-1]) * d - 0.5 * (py[1:] + py[:-1]) * v
    Rv = Rv - _zpad(0.5 * (H[1:] + H[:-1]) * (S[:-1] - S[1:]) * d, 0, 0, 1, 1)
    ui, vi = u[:, 1:-1], v[1:-1]
    qx = _zpad(0.5 * (H[:, 1:] + H[:, :-1]) * ui - 0.5 * ui.abs() * (H[:, 1:] - H[:, :-1]), 1, 1, 0, 0)
    qy = _zpad(0.5 * (H[1:] + H[:-1]) * vi - 0.5 * vi.abs() * (H[:-1] - H[1:]), 0, 0, 1, 1)
    RH = H / DT + CALV * (1 - g) * H + (qx[:, 1:] - qx[:, :-1] + qy[:-1] - qy[1:]) * d
    return Ru, Rv, RH


def _cell_context(s, dx, u, v, H):
    """What a cell's local problem sees of its neighbours: the viscosity and
    the state at the start of the sweep."""
    ny, nx = H.shape
    c = {"eta": _eta(s, u, v, dx), "H": H, "bed": s["bed"], "beta": s["beta"], "g": _sig(s["bed"] + RR * H)}
    n = {k: {o: _cl(a, *o) for o in [(a_, b_) for a_ in (-1, 0, 1) for b_ in (-1, 0, 1)]} for k, a in c.items()}
    ul, vt = u[:, :-1], v[:-1]
    cu = lambda di, dj: u[torch.arange(ny, device=u.device).add(di).clamp(0, ny - 1)][  # noqa: E731
        :, torch.arange(nx, device=u.device).add(dj).clamp(0, nx)]
    cv = lambda di, dj: v[torch.arange(ny, device=u.device).add(di).clamp(0, ny)][  # noqa: E731
        :, torch.arange(nx, device=u.device).add(dj).clamp(0, nx - 1)]
    ok = torch.ones(ny, nx, device=u.device, dtype=u.dtype)
    val = {"l": ok.clone(), "r": ok.clone(), "t": ok.clone(), "b": ok.clone()}
    val["l"][:, 0] = 0
    val["r"][:, -1] = 0
    val["t"][0] = 0
    val["b"][-1] = 0
    return dict(n=n, cu=cu, cv=cv, val=val, d=1.0 / dx, x0=(ul, u[:, 1:], vt, v[1:], H))


def _cell_rows(c, f, x):
    """The five residual rows (u_l, u_r, v_t, v_b, H) of every cell for its own
    unknowns x, all else frozen; f: the right-hand sides of those rows."""
    ul, ur, vt, vb, H = x
    n, cu, cv, w, d = c["n"], c["cu"], c["cv"], c["val"], c["d"]
    eta, Hn, bed, beta, g = n["eta"], n["H"], n["bed"], n["beta"], n["g"]
    o, L, R, T, B = (0, 0), (0, -1), (0, 1), (-1, 0), (1, 0)
    gc = _sig(bed[o] + RR * H).detach()
    eH = {k: eta[k] * Hn[k] for k in eta}
    eH[o] = eta[o] * H
    ux, vy = (ur - ul) * d, (vt - vb) * d
    sxx, syy = 2 * eH[o] * (2 * ux + vy), 2 * eH[o] * (ux + 2 * vy)
    sl = 2 * eH[L] * (2 * (ul - cu(0, -1)) + cv(0, -1) - cv(1, -1)) * d * w["l"]
    sr = 2 * eH[R] * (2 * (cu(0, 2) - ur) + cv(0, 1) - cv(1, 1)) * d * w["r"]
    st = 2 * eH[T] * (cu(-1, 1) - cu(-1, 0) + 2 * (cv(-1, 0) - vt)) * d * w["t"]
    sb = 2 * eH[B] * (cu(1, 1) - cu(1, 0) + 2 * (vb - cv(2, 0))) * d * w["b"]
    q = lambda *k: 0.25 * sum(eH[i] for i in k)  # noqa: E731
    # a corner's shear stress enters the local matrix through the row's own kind of face only
    def corners(ul, ur, vt, vb):
        return (q(o, L, T, (-1, -1)) * (cu(-1, 0) - ul + vt - cv(0, -1)) * d * w["t"] * w["l"],
                q(o, R, T, (-1, 1)) * (cu(-1, 1) - ur + cv(0, 1) - vt) * d * w["t"] * w["r"],
                q(o, L, B, (1, -1)) * (ul - cu(1, 0) + vb - cv(1, -1)) * d * w["b"] * w["l"],
                q(o, R, B, (1, 1)) * (ur - cu(1, 1) + cv(1, 1) - vb) * d * w["b"] * w["r"])

    tl, tr, bl, br = corners(ul, ur, vt.detach(), vb.detach())
    vtl, vtr, vbl, vbr = corners(ul.detach(), ur.detach(), vt, vb)
    be = {k: g[k] * beta[k] + (1 - g[k]) * DRAG for k in (L, R, T, B)}
    bc = gc * beta[o] + (1 - gc) * DRAG
    S = {k: _surf(bed[k], Hn[k]) for k in (L, R, T, B)}
    Sc = _surf(bed[o], H)
    drive = lambda k, sgn, wk: 0.5 * (H + Hn[k]) * sgn * (Sc - S[k]) * d * wk  # noqa: E731
    flux = lambda vel, a, b, wk: (0.5 * (a + b) * vel - 0.5 * vel.abs() * (b - a)) * wk  # noqa: E731
    r0 = (sxx - sl + tl - bl) * d - 0.5 * (be[L] + bc) * ul - drive(L, 1, w["l"]) - f[0]
    r1 = (sr - sxx + tr - br) * d - 0.5 * (be[R] + bc) * ur - drive(R, -1, w["r"]) - f[1]
    r2 = (st - syy + vtr - vtl) * d - 0.5 * (be[T] + bc) * vt - drive(T, -1, w["t"]) - f[2]
    r3 = (syy - sb + vbr - vbl) * d - 0.5 * (be[B] + bc) * vb - drive(B, 1, w["b"]) - f[3]
    r4 = H / DT + CALV * (1 - gc) * H - f[4]
    r4 = r4 + (flux(ur, H, Hn[R], w["r"]) - flux(ul, Hn[L], H, w["l"]) + flux(vt, H, Hn[T], w["t"]) -
               flux(vb, Hn[B], H, w["b"])) * d
    return torch.stack([r0, r1, r2, r3, r4])


def _cell_system(c, f, x):
    """Residual rows (5, ny, nx) and local Jacobians (5, 5, ny, nx)."""
    xs = [t.detach().expand(5, *t.shape).clone().requires_grad_() for t in x]
    with torch.enable_grad():
        r = _cell_rows(c, f, xs)               # (row, copy, ny, nx): copy k differentiates row k
        J = torch.autograd.grad(sum(r[k, k].sum() for k in range(5)), xs)
    return r[:, 0].detach(), torch.stack(J, 1)


def _solve5(J, r):
    return torch.linalg.solve(J.permute(2, 3, 0, 1), r.permute(1, 2, 0).unsqueeze(-1)).squeeze(-1).permute(2, 0, 1)


def _face_f(fu, fv, fH):
    return (fu[:, :-1], fu[:, 1:], fv[:-1], fv[1:], fH)


def _active_row(J, r, H):
    """Cells whose mass balance would end below the limit hold H = limit."""
    on = (H - DT * r[4]) <= THK
    J[4] = torch.where(on, torch.zeros_like(J[4]), J[4])
    J[4, 4] = torch.where(on, torch.ones_like(J[4, 4]), J[4, 4])
    r[4] = torch.where(on, H - THK, r[4])


def _add_faces(u, v, a, du_l, du_r, dv_t, dv_b):
    u[:, :-1] += a * du_l
    u[:, 1:] += a * du_r
    v[:-1] += a * dv_t
    v[1:] += a * dv_b


def _exact_smooth(case, s):
    dx, f = case["dx"], _face_f(s["fu"], s["fv"], s["fH"])
    u, v, H = s["u"].clone(), s["v"].clone(), s["H"].clone()
    for _ in range(case["sweeps"]):
        c = _cell_context(s, dx, u.clone(), v.clone(), H.clone())
        x = list(c["x0"])
        for _ in range(case["newton"]):
            r, J = _cell_system(c, f, x)
            _active_row(J, r, x[4])
            for k in range(4):
                J[k, k] -= case["shift"]
            J[4, 4] += case["shift"]
            z = _solve5(J, r)
            x = [a - case["step"] * b for a, b in zip(x, z)]
            x[4] = x[4].clamp(min=THK)
        dl = [a - b for a, b in zip(x, c["x0"])]
        _add_faces(u, v, 0.25, *dl[:4])
        H += 0.5 * dl[4]
    return [u, v, H]


def _jvp(s, dx, U, d):
    return torch.func.jvp(lambda *a: _operator(s, dx, *a), tuple(U), tuple(d))[1]


def _exact_linear(case, s):
    dx, U = case["dx"], (s["u"], s["v"], s["H"])
    f = (s["fu"], s["fv"], s["fH"])
    r0 = [a - b for a, b in zip(_operator(s, dx, *U), f)]
    c = _cell_context(s, dx, *U)
    r, J = _cell_system(c, _face_f(*f), c["x0"])
    _active_row(J, r, s["H"])
    lu, piv = torch.linalg.lu_factor(J.permute(2, 3, 0, 1))
    d = [torch.zeros_like(a) for a in U]
    for k in range(case["sweeps"]):
        rho = r0 if k == 0 else [a + b for a, b in zip(r0, _jvp(s, dx, U, d))]
        rows = torch.stack(_face_f(*rho), -1).unsqueeze(-1)
        x = -torch.linalg.lu_solve(lu, piv, rows).squeeze(-1).permute(2, 0, 1)
        dH = torch.maximum(x[4], THK - s["H"] - d[2])
        _add_faces(d[0], d[1], 0.25, x[0], x[1], x[2], x[3])
        d[2] += 0.5 * dH
    return d


def _pull(s, dx, U, lam, m):
    """lam^T J with the rows of the cells in m replaced by the identity."""
    U = [a.detach().requires_grad_() for a in U]
    with torch.enable_grad():
        R = _operator(s, dx, *U)
        tot = (R[0] * lam[0]).sum() + (R[1] * lam[1]).sum() + (R[2] * lam[2] * (1 - m)).sum()
        o = list(torch.autograd.grad(tot, U))
    o[2] = o[2] + lam[2] * m
    return o


def _exact_adjoint_smooth(case, s):
    dx, U = case["dx"], (s["u"], s["v"], s["H"])
    m = (s["H"] <= THK + 0.1).double()
    c = _cell_context(s, dx, *U)
    _, J = _cell_system(c, _face_f(0 * s["u"], 0 * s["v"], 0 * s["H"]), c["x0"])
    J[4] = J[4] * (1 - m)
    J[4, 4] += m
    lu, piv = torch.linalg.lu_factor(J.permute(2, 3, 1, 0))
    lam = [torch.zeros_like(a) for a in U]
    par = (torch.arange(m.shape[0], device="cuda")[:, None] + torch.arange(m.shape[1], device="cuda")[None, :]) % 2
    for k in range(2 * case["sweeps"]):
        p = _pull(s, dx, U, lam, m)
        rows = torch.stack(_face_f(*[a - b for a, b in zip((s["lu"], s["lv"], s["lH"]), p)]), -1).unsqueeze(-1)
        x = torch.linalg.lu_solve(lu, piv, rows).squeeze(-1).permute(2, 0, 1) * (par == k % 2)
        _add_faces(lam[0], lam[1], 0.5, x[0], x[1], x[2], x[3])
        lam[2] += x[4]
    return lam


def _conv64(x, W, b):
    w = W.to(torch.bfloat16).double().view(W.shape[0], 3, 3, -1).permute(0, 3, 1, 2)   # the products' operand type
    return torch.relu(F.conv2d(x, w, b.double(), padding=1))


def _exact_guess(s):
    sd = torch.load("glide_b200/guess_weights.pt", map_location="cuda")
    x = torch.stack([s["H"] / 1000.0, s["bed"] / 1000.0, (torch.log(s["beta"]) + 2.2) / 0.7, s["B"] / 35.0])[None]
    x = F.pad(x, (0, 0, 0, 0, 0, 4))
    i, skips = 0, []

    def pair(x, i):
        for k in (i, i + 1):
            x = _conv64(x, sd["ws.%d" % k], sd["bs.%d" % k])
        return x, i + 2

    for k in range(4):
        x, i = pair(x, i)
        if k < 3:
            skips.append(x)
            x = F.avg_pool2d(x, 2)
    for k in (2, 1, 0):
        x = torch.cat([x.repeat_interleave(2, 2).repeat_interleave(2, 3), skips[k]], 1)
        x, i = pair(x, i)
    p = torch.einsum("oc,bcyx->oyx", sd["head_w"].double(), x) + sd["head_b"].double()[:, None, None]
    uc, vc = p[0] * VEL, p[1] * VEL
    return [torch.cat([uc[:, :1], 0.5 * (uc[:, 1:] + uc[:, :-1]), uc[:, -1:]], 1),
            torch.cat([vc[:1], 0.5 * (vc[1:] + vc[:-1]), vc[-1:]], 0)]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("forward", "adjoint"):
        return None    # whole V-cycles
    if kind == "conv_train":
        x, W, b, gy = _conv_inputs(case, seed)
        xd, Wd, bd = (t.double().requires_grad_() for t in (x, W, b))
        with torch.enable_grad():
            y = _conv64(xd.permute(0, 3, 1, 2), Wd, bd).permute(0, 2, 3, 1)
            g = torch.autograd.grad(y, (xd, Wd, bd), gy.double())
        return [y.detach(), *g]
    s = _scene(case, seed)
    if kind == "guess":
        with torch.no_grad():
            return _exact_guess(s)
    # the inputs as the level holds them
    s = {k: a.to(DTYPES[case["dtype"]]).double() for k, a in s.items()}
    if kind == "residual":
        r = [a - b for a, b in zip(_operator(s, case["dx"], s["u"], s["v"], s["H"]), (s["fu"], s["fv"], s["fH"]))]
        h = s["H"] - float(torch.tensor(THK, dtype=DTYPES[case["dtype"]]))
        fb = r[2] + h - torch.sqrt(r[2] ** 2 + h ** 2)
        return [*r, torch.stack([(a ** 2).sum() for a in (r[0], r[1], fb)])]
    if kind == "gradient":
        m = (s["H"] <= THK + 0.1).double()
        lam, U, beta = (s["lu"], s["lv"], s["lH"]), (s["u"], s["v"], s["H"]), s["beta"].clone().requires_grad_()
        R = _operator(s, case["dx"], *U, beta=beta)
        gb, = torch.autograd.grad((R[0] * lam[0]).sum() + (R[1] * lam[1]).sum(), beta)
        return [*_pull(s, case["dx"], U, lam, m), gb]
    return {"smooth": _exact_smooth, "linear": _exact_linear, "adjoint_smooth": _exact_adjoint_smooth}[kind](case, s)
