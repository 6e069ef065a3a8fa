// One cell's local Vanka problem in arrow form and its solution (terms of
// glide/cuda/vanka.cu:56-404): the march of the forward sweeps, the stored systems of
// the linear sweeps and the adjoint smoother.
#pragma once
#include "glide_common.cuh"

namespace glide {

// --------------------------------------------------------------------------
// Pairs.  The four faces of a cell are held as two pairs, (left, top) and
// (right, bottom); in FP32 a pair is one operand of Blackwell's paired
// instructions.
// --------------------------------------------------------------------------
template <typename T> struct Two {
    T x, y;
};
template <typename T> __device__ __forceinline__ Two<T> two(T x, T y) { return Two<T>{x, y}; }
template <typename T> __device__ __forceinline__ Two<T> both(T x) { return Two<T>{x, x}; }
template <typename T> __device__ __forceinline__ Two<T> operator+(Two<T> a, Two<T> b) {
    return Two<T>{a.x + b.x, a.y + b.y};
}
template <typename T> __device__ __forceinline__ Two<T> operator*(Two<T> a, Two<T> b) {
    return Two<T>{a.x * b.x, a.y * b.y};
}
template <typename T> __device__ __forceinline__ Two<T> fma2(Two<T> a, Two<T> b, Two<T> c) {
    return Two<T>{a.x * b.x + c.x, a.y * b.y + c.y};
}
template <> __device__ __forceinline__ Two<float> operator+(Two<float> a, Two<float> b) {
    const float2 r = __fadd2_rn(make_float2(a.x, a.y), make_float2(b.x, b.y));
    return Two<float>{r.x, r.y};
}
template <> __device__ __forceinline__ Two<float> operator*(Two<float> a, Two<float> b) {
    const float2 r = __fmul2_rn(make_float2(a.x, a.y), make_float2(b.x, b.y));
    return Two<float>{r.x, r.y};
}
template <> __device__ __forceinline__ Two<float> fma2(Two<float> a, Two<float> b, Two<float> c) {
    const float2 r = __ffma2_rn(make_float2(a.x, a.y), make_float2(b.x, b.y), make_float2(c.x, c.y));
    return Two<float>{r.x, r.y};
}

// --------------------------------------------------------------------------
// One cell's local problem (terms of glide/cuda/vanka.cu:56-404).  Everything
// that depends on neighbour values only (fixed during a cell's iterations) is
// evaluated once.  The unknowns are the four face velocities counted outward
// (-u_l, u_r, v_t, -v_b) and the thickness: counted outward all four faces and
// all four corners have the same formulas with the same signs.  Pairs: 1 = (left, top),
// 2 = (right, bottom); corners: p = (top left, bottom right),
// q = (bottom left, top right).
// --------------------------------------------------------------------------
template <typename T> struct Cell {
    T E;                    // 2 eta/dx^2
    Two<T> ew_p, ew_q;      // eta/(4 dx^2) at the corners (0 on the boundary)
    Two<T> S_p, S_q;        // the three neighbours' part of eta*H/dx^2 at the corners
    Two<T> X_p, X_q;        // 2 dx * shear rate of the corners at the state, signed so that outward flow adds
    Two<T> D0;              // u_r - u_l, v_t - v_b at the state
    Two<T> K_1, K_2;        // normal-stress coefficients of the four neighbours
    Two<T> B_1, B_2;        // half of the neighbours' effective drag
    Two<T> n_1, n_2;        // outward velocities at the state
    Two<T> H_1, H_2;        // neighbour thickness
    Two<T> Z_1, Z_2;        // minus the neighbour surface
    Two<T> W_1, W_2;        // -1/(2 dx) on interior faces, 0 on boundary faces
    T bed, beta, f_H, thk;
};

// The 5x5 system of one Newton step, (-J) x = -r in the velocity rows, in
// arrow form: with a = x_l + x_r and b = x_t + x_b (outward),
//   D x + p2 (2a + b) + c h   in rows l, r,
//   D x + p2 (a + 2b) + c h   in rows t, b
// (the cell's own viscous block is symmetric and of rank two,
// glide/cuda/vanka.cu:117-152) and -e . x + j4 h in the mass row, which is
// kept at half its size so that the face weights W serve the driving stress
// and the flux.  c and q are without the cell's own normal stresses sxy and
// their thickness derivatives hxy, which are common to both faces of a pair.
template <typename T> struct Arrow {
    Two<T> D1, D2, c1, c2, e1, e2, hxy;
    T p2, j4;
};

// The part of the solution that does not depend on the right-hand side.
template <typename T> struct ArrowInv {
    Two<T> i, w1, w2, Cd, k, e;
    T b11, b12, b22, ag, bg, ih;
};

// Elimination by sums and differences: the difference of a pair's rows is free
// of the own stresses and gives a D-weighted mean of the pair, the D-weighted
// sums form a 2x2 system for (a, b) whose determinant is a sum of terms of one
// sign, and the mass row gives the thickness.  Four reciprocals (two of them
// independent) instead of the five successive pivots of an unstructured 5x5
// elimination, and no subtraction of nearly equal pivots; a row with D = 0 is
// fine as long as its pair's sum is not 0.  The determinant is taken in units of
// the two pair sums: a product of two drags leaves FP32's range from 2e19 on,
// their quotients do not.  IEEE: correctly rounded reciprocals
// also in FP32 (the adjoint, whose systems are not iterated on), else M<T>::rcp
// as the forward Newton steps and the linear factors take it.
template <bool IEEE, typename T> __device__ __forceinline__ T reciprocal(T x) {
    if constexpr (IEEE)
        return T(1) / x;
    else
        return M<T>::rcp(x);
}
template <bool IEEE = false, typename T>
__device__ __forceinline__ void arrow_factor(const Arrow<T>& s, ArrowInv<T>& q) {
    const Two<T> ds = s.D1 + s.D2;
    q.i = two(reciprocal<IEEE>(ds.x), reciprocal<IEEE>(ds.y));
    q.w1 = s.D1 * q.i;
    q.w2 = s.D2 * q.i;
    const Two<T> w = q.w1 * q.w2, t = both(s.p2) * q.i, a = fma2(both(T(2)), t, w);
    const T id = reciprocal<IEEE>(w.x * a.y + t.x * (T(3) * t.y + T(2) * w.y));
    const Two<T> n = q.i * both(id);
    q.b11 = a.x * n.y;
    q.b22 = a.y * n.x;
    q.b12 = t.x * n.y;
    const Two<T> g = fma2(s.c1, q.w2, fma2(s.c2, q.w1, s.hxy));
    q.ag = q.b22 * g.x - q.b12 * g.y;
    q.bg = q.b11 * g.y - q.b12 * g.x;
    q.Cd = fma2(s.c2, both(T(-1)), s.c1);
    q.k = fma2(s.e2, both(T(-1)), s.e1) * q.i;
    q.e = fma2(s.e1, q.w2, s.e2 * q.w1);
    const Two<T> m = fma2(q.k, q.Cd, q.e * two(q.ag, q.bg));
    q.ih = reciprocal<IEEE>(s.j4 + (m.x + m.y));
}

template <typename T>
__device__ __forceinline__ void arrow_solve(const ArrowInv<T>& q, Two<T> q1, Two<T> q2, Two<T> sxy, T r4, Two<T>& x1,
                                            Two<T>& x2, T& h) {
    const Two<T> r = fma2(q1, q.w2, fma2(q2, q.w1, sxy));
    const Two<T> Qd = fma2(q2, both(T(-1)), q1);
    const Two<T> ar = two(q.b22 * r.x - q.b12 * r.y, q.b11 * r.y - q.b12 * r.x);
    const Two<T> t = fma2(q.k, Qd, q.e * ar);
    h = (r4 + (t.x + t.y)) * q.ih;
    const Two<T> hn = both(-h);
    const Two<T> ab = fma2(two(q.ag, q.bg), hn, ar);
    const Two<T> m = fma2(q.Cd, hn, Qd) * q.i;
    x1 = fma2(q.w2, ab, m);
    x2 = fma2(q.w1, ab, m * both(T(-1)));
}

template <typename T> __device__ __forceinline__ bool neg(T x);   // sign bit, as copysign sees it
template <> __device__ __forceinline__ bool neg<float>(float x) { return __float_as_int(x) < 0; }
template <> __device__ __forceinline__ bool neg<double>(double x) { return __double2hiint(x) < 0; }

// The matrix at the cell's state.  active: -1 tests H - dt r_H <= gamma
// (vanka.cu:104-113), 0 / 1 force the row; shift: vanka.cu:406-410.
template <typename T>
__device__ __forceinline__ void arrow_assemble(const Cell<T>& C, T h, T shift, int active, const Phys<T>& p,
                                               Arrow<T>& s) {
    const T rr = rho_ratio<T>(), hdti = T(0.5) / p.dt;
    const T g = sigmoid(C.bed + rr * h, p.sig_c);
    const Two<T> hh = both(h);
    // own normal stresses
    {
        const Two<T> e = C.D0 + both(C.D0.x + C.D0.y);
        s.p2 = C.E * h;
        s.hxy = both(C.E) * e;
    }
    // neighbours' normal stresses, basal drag
    {
        const T bc = T(0.5) * (p.water_drag + g * (C.beta - p.water_drag));
        s.D1 = (C.K_1 + both(shift)) + (C.B_1 + both(bc));
        s.D2 = (C.K_2 + both(shift)) + (C.B_2 + both(bc));
    }
    // corner shear stresses: a corner's stress enters the rows of its two faces
    {
        const Two<T> Gp = fma2(C.ew_p, hh, C.S_p), Gq = fma2(C.ew_q, hh, C.S_q);
        const Two<T> ep = C.ew_p * C.X_p, eq = C.ew_q * C.X_q;
        s.D1 = s.D1 + two(Gp.x + Gq.x, Gp.x + Gq.y);
        s.D2 = s.D2 + two(Gp.y + Gq.y, Gp.y + Gq.x);
        s.c1 = two(ep.x + eq.x, ep.x + eq.y);
        s.c2 = two(ep.y + eq.y, ep.y + eq.x);
    }
    if (p.gl_deriv) {
        const Two<T> dg = both(T(0.5) * rr * (p.sig_c * g * (T(1) - g)) * (C.beta - p.water_drag));
        s.c1 = fma2(dg, C.n_1, s.c1);
        s.c2 = fma2(dg, C.n_2, s.c2);
    }
    // driving stress
    {
        const bool fl = !(C.bed > -rr * h);
        const Two<T> Z = both((fl ? -rr * h : C.bed) + h), k = both(fl ? T(1) - rr : T(1));
        s.c1 = fma2(C.W_1 * (C.H_1 + hh), k, fma2(C.W_1, Z + C.Z_1, s.c1));
        s.c2 = fma2(C.W_2 * (C.H_2 + hh), k, fma2(C.W_2, Z + C.Z_2, s.c2));
    }
    // half of the mass row: upwind fluxes, calving (flux.cu:39-64, :187-211)
    {
        const T cal = T(0.5) * p.calving_rate * (T(1) - g);
        // inward by the sign bit, a zero's too (copysign, flux.cu:53): the neighbour's thickness
        s.e1 = C.W_1 * two(neg(C.n_1.x) ? C.H_1.x : h, neg(C.n_1.y) ? C.H_1.y : h);
        s.e2 = C.W_2 * two(neg(C.n_2.x) ? C.H_2.x : h, neg(C.n_2.y) ? C.H_2.y : h);
        const Two<T> o = fma2(C.W_1, two(M<T>::max(C.n_1.x, T(0)), M<T>::max(C.n_1.y, T(0))),
                              C.W_2 * two(M<T>::max(C.n_2.x, T(0)), M<T>::max(C.n_2.y, T(0))));
        s.j4 = (hdti + cal) - (o.x + o.y);
        if (p.gl_deriv) s.j4 -= T(0.5) * p.calving_rate * h * (rr * (p.sig_c * g * (T(1) - g)));
        bool on = active > 0;
        if (active < 0) {
            const Two<T> t = fma2(s.e1, C.n_1, s.e2 * C.n_2);
            const T r4 = h * (hdti + cal) - T(0.5) * C.f_H - (t.x + t.y);
            on = (h - p.dt * (T(2) * r4)) <= C.thk;
        }
        if (on) {
            s.e1 = s.e2 = both(T(0));
            s.j4 = T(0.5);
        }
        s.j4 += T(0.5) * shift;
    }
}

// J^T x = b of one cell in the arrow form: the velocity block is symmetric, the
// thickness column and the mass row change places (the mass row is stored at
// half its size).
template <typename T> __device__ __forceinline__ Arrow<T> transposed(const Arrow<T>& s) {
    Arrow<T> t = s;
    t.c1 = s.e1 + s.e1;
    t.c2 = s.e2 + s.e2;
    t.e1 = s.c1 + two(s.hxy.x, s.hxy.y);
    t.e2 = s.c2 + two(s.hxy.x, s.hxy.y);
    t.hxy = both(T(0));
    t.j4 = T(2) * s.j4;
    return t;
}

// lambda += omega * (half of each face's change, the full thickness change);
// within one colour every face has one writer
template <bool CHAIN, typename T>
__device__ __forceinline__ void adjoint_update(const ArrowInv<T>& q, const T* __restrict__ ra_u,
                                               const T* __restrict__ ra_v, const T* __restrict__ ra_H,
                                               T* __restrict__ l_u, T* __restrict__ l_v, T* __restrict__ l_H, int i,
                                               int j, int nx, T omega) {
    const int iu = i * (nx + 1) + j, ic = i * nx + j;
    Two<T> x1, x2;
    T xh;
    arrow_solve(q, two(ld<CHAIN>(ra_u + iu), -ld<CHAIN>(ra_v + ic)),
                two(-ld<CHAIN>(ra_u + iu + 1), ld<CHAIN>(ra_v + ic + nx)), both(T(0)), ld<CHAIN>(ra_H + ic), x1, x2, xh);
    l_u[iu] -= T(0.5) * omega * x1.x;
    l_u[iu + 1] += T(0.5) * omega * x2.x;
    l_v[ic] += T(0.5) * omega * x1.y;
    l_v[ic + nx] -= T(0.5) * omega * x2.y;
    l_H[ic] += omega * xh;
}

// What the sweeps with stored systems read, one array of nc cells after the
// other: the matrix for the linear sweep, the solved form for the adjoint.
constexpr int LU_N = 14;    // D1, D2, p2, c1, c2, e1, e2, j4
constexpr int LU_ROOM = 25; // arrays per problem in the caller's buffer
constexpr int ADJ_N = 18;   // i, w1, w2, Cd, k, e, b11, b12, b22, ag, bg, ih
template <typename T> __device__ __forceinline__ void store_matrix(T* out, int64_t nc, const Arrow<T>& s) {
    const Two<T> c1 = s.c1 + s.hxy, c2 = s.c2 + s.hxy;
    const T o[LU_N] = {s.D1.x, s.D1.y, s.D2.x, s.D2.y, s.p2, c1.x, c1.y, c2.x, c2.y, s.e1.x, s.e1.y,
                       s.e2.x, s.e2.y, s.j4};
#pragma unroll
    for (int k = 0; k < LU_N; k++) out[k * nc] = o[k];
}
template <typename T> __device__ __forceinline__ void store_solved(T* out, int64_t nc, const ArrowInv<T>& q) {
    const T o[ADJ_N] = {q.i.x, q.i.y, q.w1.x, q.w1.y, q.w2.x, q.w2.y, q.Cd.x, q.Cd.y, q.k.x,
                        q.k.y, q.e.x, q.e.y, q.b11, q.b12, q.b22, q.ag, q.bg, q.ih};
#pragma unroll
    for (int k = 0; k < ADJ_N; k++) out[k * nc] = o[k];
}

// Which cells' systems a kernel forms, and what becomes of them.
enum { STORE_LU = 0, STORE_ADJOINT = 1, SOLVE_ADJOINT = 2 };
template <typename T> struct StoredArgs {
    const T *u, *v, *H, *f_H, *bed, *B, *beta, *gamma;
    const T* act;               // active set; null: tested with f_H
    T* out;                     // stored arrays
    T shift;
    T *l_u, *l_v, *l_H;         // SOLVE_ADJOINT: multiplier, adjoint residual, colour
    const T *ra_u, *ra_v, *ra_H;
    T omega;
    int color;
    int n_strips, rows, n_warps;   // march
    int y0;                        // tile
};

}  // namespace glide
