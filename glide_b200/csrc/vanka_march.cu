// Forward Vanka cell kernel, marching form with the arrow-form local solve
// (cell_system.cuh); writes the same five cell arrays as vanka_cells_kernel
// (vanka.cu), which vanka_apply_kernel turns into the update of U.
//
// A warp owns 30 cell columns and marches down a chunk of rows with the rows
// in reach in registers and the neighbouring columns in its lanes: every
// viscosity, grounded fraction, surface and drag is computed once per launch
// and every field read once per row, where a thread per cell of a tile takes
// five sigmoids and a ring of viscosities; 30 cells with 10 Newton steps are 2,590
// warp instructions (32 cells of the tile form 4,870), with four reciprocals a
// step (two of them independent) instead of five successive pivots.  The unknowns are the
// increments of the face velocities over their values at the start, so the
// differences of nearby velocities that the strain rates need are formed once,
// from the unrounded state.
//
// What bounds it: instruction issue and the latency of a step's chain at the 13
// (FP64: 8) warps that an SM's registers hold; FP32, 1024^2, 10 steps: issue slots
// 62 % active, FMA pipe 43 %, DRAM 4 %.  Figures of both forms: use_march in
// vanka.cu.
#include <type_traits>

#include "cell_system.cuh"

namespace glide {

constexpr int SW = 30;          // cell columns per warp
constexpr int VC_NT = 128;
// Resident CTAs per SM asked of the compiler: 128 registers a thread in FP32, 255
// in FP64.  1024^2, 10 Newton steps: FP32 5 CTAs 151 us per sweep, 4 136; FP64 3
// CTAs 341, 2 348, but 256^2 with 2 steps 14.9 against 12.5.
template <typename T> constexpr int VC_CTAS = sizeof(T) == 4 ? 4 : 2;
constexpr int REF_STRIDE = 14;  // reference block stride (glide/grid.py:182-188)

template <bool CHAIN> __device__ __forceinline__ bool tile_on(const int* flags, int i, int j, int nx) {
    return ld<CHAIN>(flags + (i / REF_STRIDE) * (nx / REF_STRIDE + 1) + j / REF_STRIDE) != 0;
}

// Matrix and residual at the iterate (n + d, h); R: minus the residual terms
// that stay fixed (neighbour stresses at the start, f).
template <typename T>
__device__ __forceinline__ void newton_assemble(const Cell<T>& C, Two<T> R1, Two<T> R2, Two<T> d1, Two<T> d2, T h,
                                                T hdti, T shift, const Phys<T>& p, Arrow<T>& s, Two<T>& q1,
                                                Two<T>& q2, Two<T>& sxy, T& r4) {
    const T rr = rho_ratio<T>();
    const T g = sigmoid(C.bed + rr * h, p.sig_c);
    const Two<T> n1 = C.n_1 + d1, n2 = C.n_2 + d2, hh = both(h);
    // own normal stresses
    {
        const Two<T> d = C.D0 + (d1 + d2);
        const Two<T> e = d + both(d.x + d.y);
        s.p2 = C.E * h;
        sxy = both(s.p2) * e;
        s.hxy = both(C.E) * e;
    }
    // neighbours' normal stresses, basal drag
    {
        const T bc = T(0.5) * (p.water_drag + g * (C.beta - p.water_drag));
        const Two<T> b1 = C.B_1 + both(bc), b2 = C.B_2 + both(bc);
        q1 = fma2(b1, n1, fma2(C.K_1, d1, R1));
        q2 = fma2(b2, n2, fma2(C.K_2, d2, R2));
        s.D1 = (C.K_1 + both(shift)) + b1;
        s.D2 = (C.K_2 + both(shift)) + b2;
    }
    // corner shear stresses: a corner's stress enters the rows of its two faces
    {
        const Two<T> Gp = fma2(C.ew_p, hh, C.S_p), Gq = fma2(C.ew_q, hh, C.S_q);
        const Two<T> Xp = C.X_p + two(d1.x + d1.y, d2.x + d2.y), Xq = C.X_q + two(d1.x + d2.y, d2.x + d1.y);
        const Two<T> tp = Gp * Xp, tq = Gq * Xq, ep = C.ew_p * Xp, eq = C.ew_q * Xq;
        q1 = q1 + two(tp.x + tq.x, tp.x + tq.y);
        q2 = q2 + two(tp.y + tq.y, tp.y + tq.x);
        s.D1 = s.D1 + two(Gp.x + Gq.x, Gp.x + Gq.y);
        s.D2 = s.D2 + two(Gp.y + Gq.y, Gp.y + Gq.x);
        s.c1 = two(ep.x + eq.x, ep.x + eq.y);
        s.c2 = two(ep.y + eq.y, ep.y + eq.x);
    }
    if (p.gl_deriv) {
        const Two<T> dg = both(T(0.5) * rr * (p.sig_c * g * (T(1) - g)) * (C.beta - p.water_drag));
        s.c1 = fma2(dg, n1, s.c1);
        s.c2 = fma2(dg, n2, s.c2);
    }
    // driving stress
    {
        const bool fl = !(C.bed > -rr * h);
        const Two<T> Z = both((fl ? -rr * h : C.bed) + h), k = both(fl ? T(1) - rr : T(1));
        Two<T> w = C.W_1 * (C.H_1 + hh), z = Z + C.Z_1;
        q1 = fma2(w, z, q1);
        s.c1 = fma2(w, k, fma2(C.W_1, z, s.c1));
        w = C.W_2 * (C.H_2 + hh);
        z = Z + C.Z_2;
        q2 = fma2(w, z, q2);
        s.c2 = fma2(w, k, fma2(C.W_2, z, s.c2));
    }
    // half of the mass row: upwind fluxes, calving (flux.cu:39-64, :187-211)
    {
        const T cal = T(0.5) * p.calving_rate * (T(1) - g);
        // inward by the sign bit, a zero's too (copysign, flux.cu:53): the neighbour's thickness
        s.e1 = C.W_1 * two(neg(n1.x) ? C.H_1.x : h, neg(n1.y) ? C.H_1.y : h);
        s.e2 = C.W_2 * two(neg(n2.x) ? C.H_2.x : h, neg(n2.y) ? C.H_2.y : h);
        const Two<T> t = fma2(s.e1, n1, s.e2 * n2);
        r4 = h * (hdti + cal) - T(0.5) * C.f_H - (t.x + t.y);
        const Two<T> o = fma2(C.W_1, two(M<T>::max(n1.x, T(0)), M<T>::max(n1.y, T(0))),
                              C.W_2 * two(M<T>::max(n2.x, T(0)), M<T>::max(n2.y, T(0))));
        s.j4 = (hdti + cal) - (o.x + o.y);
        if (p.gl_deriv) s.j4 -= T(0.5) * p.calving_rate * h * (rr * (p.sig_c * g * (T(1) - g)));
        if ((h - p.dt * (T(2) * r4)) <= C.thk) {
            s.e1 = s.e2 = both(T(0));
            s.j4 = T(0.5);
            r4 = T(0.5) * (h - C.thk);
        }
        s.j4 += T(0.5) * shift;
    }
}

template <typename T> struct MarchArgs {
    const T *u, *v, *H, *f_u, *f_v, *f_H, *bed, *B, *beta, *gamma;
    const int *flags, *any_active;
    T* out;
    int n_newton;
    T shift, step;
    int n_strips, rows, n_warps;
};

template <typename T>
__device__ __forceinline__ void newton_cell(const Cell<T>& C, Two<T> R1, Two<T> R2, T H0, int n_newton, T shift,
                                            T step, const Phys<T>& p, Two<T>& d1, Two<T>& d2, T& dh) {
    const T hdti = T(0.5) / p.dt;
    d1 = d2 = both(T(-0.0));   // x + (-0) keeps the sign of a zero velocity x
    T h = H0;
    for (int it = 0; it < n_newton; it++) {
        Arrow<T> s;
        ArrowInv<T> q;
        Two<T> q1, q2, sxy, x1, x2;
        T r4, xh;
        newton_assemble(C, R1, R2, d1, d2, h, hdti, shift, p, s, q1, q2, sxy, r4);
        arrow_factor(s, q);
        arrow_solve(q, q1, q2, sxy, r4, x1, x2, xh);
        // reference step 0.25: relaxation_factor, glide/cuda/vanka.cu:416
        d1 = fma2(both(-step), x1, d1);
        d2 = fma2(both(-step), x2, d2);
        h = M<T>::max(h - step * xh, C.thk);
    }
    dh = h - H0;
    if (!(isfinite(d1.x) && isfinite(d1.y) && isfinite(d2.x) && isfinite(d2.y) && isfinite(dh))) {
        d1 = d2 = both(T(0));  // a failed local solve leaves its cell unchanged
        dh = T(0);
    }
}

template <typename T, bool LOCAL, bool CHAIN, typename P>
__global__ void __launch_bounds__(VC_NT, VC_CTAS<T>)
    vanka_march_kernel(const MarchArgs<T> A, Geo g, P p) {
    const int zero = chain_enter<CHAIN>();
    const int ny = g.ny, nx = g.nx, b = blockIdx.y + zero;
    if (LOCAL && ld<CHAIN>(A.any_active + b) == 0) return;
    const int wid = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32 + zero;
    if (wid >= A.n_warps) return;  // whole warp
    const int lane = threadIdx.x & 31;
    const unsigned FULL = 0xffffffffu;
    const int64_t nc = g.nc();
    const T* __restrict__ u = A.u + b * g.nu();
    const T* __restrict__ v = A.v + b * g.nv();
    const T* __restrict__ H = A.H + b * nc;
    const T* __restrict__ bed = A.bed + b * nc;
    const T* __restrict__ B = A.B + b * nc;
    const T* __restrict__ beta = A.beta + b * nc;
    const T* __restrict__ gamma = A.gamma + b * nc;
    const T* __restrict__ f_u = A.f_u + b * g.nu();
    const T* __restrict__ f_v = A.f_v + b * g.nv();
    const T* __restrict__ f_H = A.f_H + b * nc;
    T* __restrict__ out = A.out + b * nc * 5;
    const int* flags = LOCAL ? A.flags + b * int64_t(ny / REF_STRIDE + 1) * (nx / REF_STRIDE + 1) : nullptr;

    const int strip = wid % A.n_strips, chunk = wid / A.n_strips;
    const int i0 = chunk * A.rows, i1 = min(i0 + A.rows, ny);
    const int jc = strip * SW - 1 + lane;
    const int jcc = clampi(jc, 0, nx - 1), juL = clampi(jc, 0, nx), juR = clampi(jc + 1, 0, nx);
    const int jvL = clampi(jc - 1, 0, nx - 1), jvR = clampi(jc + 1, 0, nx - 1);
    const bool first = lane == 0, last = lane == 31;
    const bool own = lane >= 1 && lane <= SW && jc < nx;
    if (LOCAL) {   // a chunk without an active cell does nothing
        bool any = false;
        if (own)
            for (int i = i0; i < i1 && !any; i += (i1 - 1 - i > 0 ? min(REF_STRIDE, i1 - 1 - i) : 1))
                any = tile_on<CHAIN>(flags, i, jc, nx);
        if (!__any_sync(FULL, any)) return;
    }
    const T dxi = p.dxi, d2 = p.dxi * p.dxi, rr = rho_ratio<T>();
    auto U = [&](int r, int col) -> T { return ld<CHAIN>(u + (clampi(r, 0, ny - 1) * (nx + 1) + col)); };
    auto V = [&](int r, int col) -> T { return ld<CHAIN>(v + (clampi(r, 0, ny) * nx + col)); };
    auto row = [&](const T* a, int r) -> T { return ld<CHAIN>(a + (clampi(r, 0, ny - 1) * nx + jcc)); };

    // at the start of iteration i: u rows i-1..i+1, v rows i-1..i+1, cell rows i-1 and i
    int i = i0 - 2;
    T um = T(0), u0 = U(i, juL), u1 = U(i + 1, juL);
    T uR0 = last ? U(i, juR) : T(0), uR1 = last ? U(i + 1, juR) : T(0), uRm = T(0);
    T vm = T(0), v0 = V(i, jcc), v1 = V(i + 1, jcc);
    T vL1 = first ? V(i + 1, jvL) : T(0), vR1 = last ? V(i + 1, jvR) : T(0);
    T Hm = T(0), Zm = T(0), bm = T(0), em = T(0);              // row i-1: H, surface, drag, eta*H
    T Hc = T(0), Zc = T(0), bc = T(0), ec = T(0), etac = T(0); // row i
    T bedc = T(0), betac = T(0);
    for (; i < i1; ++i) {
        const T u2 = U(i + 2, juL), uR2 = last ? U(i + 2, juR) : T(0);
        const T v2 = V(i + 2, jcc), vL2 = first ? V(i + 2, jvL) : T(0), vR2 = last ? V(i + 2, jvR) : T(0);
        const T Hp = row(H, i + 1), bedp = row(bed, i + 1), betap = row(beta, i + 1), Bp = row(B, i + 1);
        T u0r = __shfl_down_sync(FULL, u0, 1), u1r = __shfl_down_sync(FULL, u1, 1);
        T u2r = __shfl_down_sync(FULL, u2, 1);
        T v1l = __shfl_up_sync(FULL, v1, 1), v2l = __shfl_up_sync(FULL, v2, 1);
        T v1r = __shfl_down_sync(FULL, v1, 1), v2r = __shfl_down_sync(FULL, v2, 1);
        if (last) { u0r = uR0; u1r = uR1; u2r = uR2; v1r = vR1; v2r = vR2; }
        if (first) { v1l = vL1; v2l = vL2; }
        EtaIn<T> a;
        a.ul = u1;   a.ur = u1r;   a.vt = v1;   a.vb = v2;
        a.u_tl = u0; a.u_tr = u0r; a.u_bl = u2; a.u_br = u2r;
        a.v_lt = v1l; a.v_rt = v1r; a.v_lb = v2l; a.v_rb = v2r;
        const T etap = cell_eta(a, Bp, clampi(i + 1, 0, ny - 1), jcc, ny, nx, p).eta, ep = etap * Hp;
        const T Zp = M<T>::max(bedp, -rr * Hp) + Hp;
        const T gp = sigmoid(bedp + rr * Hp, p.sig_c);
        const T bp = gp * betap + (T(1) - gp) * p.water_drag;

        bool on = own;
        if (LOCAL) on = on && i >= i0 && tile_on<CHAIN>(flags, i, jc, nx);
        if (i >= i0 && (!LOCAL || __any_sync(FULL, on))) {  // warp-uniform
            Cell<T> C;
            const T wl = jc > 0 ? T(1) : T(0), wr = jc + 1 < nx ? T(1) : T(0);
            const T wt = i > 0 ? T(1) : T(0), wb = i + 1 < ny ? T(1) : T(0);
            T umr = __shfl_down_sync(FULL, um, 1);
            if (last) umr = uRm;
            const T v0l = __shfl_up_sync(FULL, v0, 1), v0r = __shfl_down_sync(FULL, v0, 1);
            const T ull = __shfl_up_sync(FULL, u0, 1), urr = __shfl_down_sync(FULL, u0r, 1);
            const T eL = __shfl_up_sync(FULL, ec, 1), eR = __shfl_down_sync(FULL, ec, 1);
            const T emL = __shfl_up_sync(FULL, em, 1), emR = __shfl_down_sync(FULL, em, 1);
            const T epL = __shfl_up_sync(FULL, ep, 1), epR = __shfl_down_sync(FULL, ep, 1);
            const T bL = __shfl_up_sync(FULL, bc, 1), bR = __shfl_down_sync(FULL, bc, 1);
            const T HL = __shfl_up_sync(FULL, Hc, 1), HR = __shfl_down_sync(FULL, Hc, 1);
            const T ZL = __shfl_up_sync(FULL, Zc, 1), ZR = __shfl_down_sync(FULL, Zc, 1);
            C.H_1 = two(HL, Hm);
            C.H_2 = two(HR, Hp);
            C.Z_1 = two(-ZL, -Zm);
            C.Z_2 = two(-ZR, -Zp);
            C.B_1 = two(T(0.5) * bL, T(0.5) * bm);
            C.B_2 = two(T(0.5) * bR, T(0.5) * bp);
            C.bed = bedc;
            C.beta = betac;
            C.n_1 = two(-u0, v0);
            C.n_2 = two(u0r, -v1);
            C.D0 = two(u0r - u0, v0 - v1);
            C.E = T(2) * d2 * etac;
            const T e4 = T(0.25) * d2 * etac, q = T(0.25) * d2;
            C.ew_p = two(e4 * wt * wl, e4 * wb * wr);
            C.ew_q = two(e4 * wb * wl, e4 * wt * wr);
            C.S_p = two(q * (emL + em + eL) * wt * wl, q * (eR + ep + epR) * wb * wr);
            C.S_q = two(q * (eL + epL + ep) * wb * wl, q * (em + emR + eR) * wt * wr);
            C.X_p = two((um - u0) + (v0 - v0l), (u0r - u1r) + (v1r - v1));
            C.X_q = two((u1 - u0) + (v1l - v1), (u0r - umr) + (v0 - v0r));
            C.K_1 = two(T(4) * d2 * eL * wl, T(4) * d2 * em * wt);
            C.K_2 = two(T(4) * d2 * eR * wr, T(4) * d2 * ep * wb);
            C.W_1 = two(T(-0.5) * dxi * wl, T(-0.5) * dxi * wt);
            C.W_2 = two(T(-0.5) * dxi * wr, T(-0.5) * dxi * wb);
            if (on) {
                const int ic = i * nx + jc, iu = i * (nx + 1) + jc;
                // minus the residual terms that stay fixed: neighbour stresses at the start, f
                const Two<T> R1 = two(-(C.K_1.x * ((u0 - ull) + T(0.5) * (v0l - v1l))) - ld<CHAIN>(f_u + iu),
                                      -(C.K_1.y * ((vm - v0) + T(0.5) * (umr - um))) + ld<CHAIN>(f_v + ic));
                const Two<T> R2 = two(-(C.K_2.x * ((urr - u0r) + T(0.5) * (v0r - v1r))) + ld<CHAIN>(f_u + iu + 1),
                                      -(C.K_2.y * ((v1 - v2) + T(0.5) * (u1r - u1))) - ld<CHAIN>(f_v + ic + nx));
                C.thk = ld<CHAIN>(gamma + ic);
                C.f_H = ld<CHAIN>(f_H + ic);
                Two<T> x1, x2;
                T dh;
                newton_cell<T>(C, R1, R2, Hc, A.n_newton, A.shift, A.step, p, x1, x2, dh);
                out[ic] = T(-0.5) * x1.x;
                out[nc + ic] = T(0.5) * x2.x;
                out[2 * nc + ic] = T(0.5) * x1.y;
                out[3 * nc + ic] = T(-0.5) * x2.y;
                out[4 * nc + ic] = dh;
            }
        }
        // roll the window one row down
        um = u0; u0 = u1; u1 = u2; uRm = uR0; uR0 = uR1; uR1 = uR2;
        vm = v0; v0 = v1; v1 = v2; vL1 = vL2; vR1 = vR2;
        Hm = Hc; Zm = Zc; bm = bc; em = ec;
        Hc = Hp; Zc = Zp; bc = bp; ec = ep; etac = etap; bedc = bedp; betac = betap;
    }
}

// Rows per warp: as few waves of resident warps as chunks of at most 32 rows
// allow, the rows spread evenly over them (a chunk's two preparatory rows cost
// about 10 % of a row of two Newton steps each).  Grids too small to fill the
// chip take one row per warp and spread the warps over all SMs.  A gated sweep
// takes one row, two beyond four waves: which rows are active is not known here,
// and only short chunks spread them over the chip (a quarter of the rows active,
// 10 Newton steps: even chunks / these at 1024^2 FP32 90.9 / 53.9 us; one row / two at
// 1024^2 FP32 60.9 / 56.7, at 256^2 FP64 21.8 / 27.8).
template <typename T>
void run_march(const GlideLevelArgs* a, const void* f_u, const void* f_v, const void* f_H, int n_newton, double shift,
               double step, const int* flags, const int* any_active, void* scratch, cudaStream_t s) {
    Geo g{a->ny, a->nx, a->nb};
    const int64_t resident = 148 * (VC_NT / 32) * VC_CTAS<T>;
    MarchArgs<T> A{};
    A.n_strips = (g.nx + SW - 1) / SW;
    const int64_t units = int64_t(A.n_strips) * g.ny * g.nb;
    const int64_t waves = (units + 32 * resident - 1) / (32 * resident);
    const int64_t rows = (units + waves * resident - 1) / (waves * resident);
    const int64_t short_chunk = units > 4 * resident ? 2 : 1;
    const int64_t most = flags && g.ny > short_chunk ? short_chunk : g.ny;
    A.rows = int(rows < most ? rows : most);
    A.n_warps = A.n_strips * ((g.ny + A.rows - 1) / A.rows);
    const int64_t per_sm = (int64_t(A.n_warps) * g.nb + 147) / 148;
    const int threads = 32 * int(per_sm < VC_NT / 32 ? per_sm : VC_NT / 32);
    const dim3 grid((A.n_warps + threads / 32 - 1) / (threads / 32), g.nb);
    A.u = (const T*)a->u; A.v = (const T*)a->v; A.H = (const T*)a->H;
    A.f_u = (const T*)f_u; A.f_v = (const T*)f_v; A.f_H = (const T*)f_H;
    A.bed = (const T*)a->bed; A.B = (const T*)a->B; A.beta = (const T*)a->beta; A.gamma = (const T*)a->gamma;
    A.flags = flags; A.any_active = any_active;
    A.out = (T*)scratch;
    A.n_newton = n_newton; A.shift = T(shift); A.step = T(step);
    with_glen(a->params, make_phys<T>(a->params, a->dx, a->dt), [&](auto p) {
        using P = decltype(p);
        auto go = [&](auto chain) {
            constexpr bool CHAIN = decltype(chain)::value;
            auto run = [&](auto kernel) { launch_chained<CHAIN>(kernel, grid, threads, s, A, g, p); };
            flags ? run(vanka_march_kernel<T, true, CHAIN, P>) : run(vanka_march_kernel<T, false, CHAIN, P>);
        };
        blocks_of(grid) <= 148 ? go(std::true_type{}) : go(std::false_type{});
    });
}
template void run_march<float>(const GlideLevelArgs*, const void*, const void*, const void*, int, double, double,
                               const int*, const int*, void*, cudaStream_t);
template void run_march<double>(const GlideLevelArgs*, const void*, const void*, const void*, int, double, double,
                                const int*, const int*, void*, cudaStream_t);

}  // namespace glide
