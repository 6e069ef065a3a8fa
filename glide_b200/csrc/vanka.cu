// Cell-patch Vanka smoothers (glide/cuda/vanka.cu) on B200.
//
// Forward sweep = two kernels:
//   the cell kernel runs the damped local Newton iterations on each cell's 5
//     unknowns (u_l, u_r, v_t, v_b, H_c) with the neighbours and the viscosity
//     frozen, and stores half of each face change and the full H change per
//     cell (deterministic, no atomics): here a thread per cell of a tile
//     (vanka_cells), in vanka_march.cu a march down rows; use_march chooses;
//   vanka_apply: every face adds the halves of its two cells, U += omega*delta
//     (the reference zero-fills a delta vector, scatters with atomicAdd and
//     axpys on the host: glide/grid.py:305-317, vanka.cu:433-437).
// In the tile form the viscosity of the tile plus a one-cell ring is computed once into shared
// memory; the neighbours' grounding sigmoids are hoisted out of the Newton
// loop.  The local variant gates cells by the reference's 16x16-window /
// stride-14 block rule (vanka.cu:875-888) through per-tile flags.
#include <type_traits>

#include "glide_common.cuh"

namespace glide {

constexpr int VX = 32;   // tile width; a tile is VX x VY cells, VY = 8, 4 or 1 (see cell_tile)
constexpr int REF_STRIDE = 14;   // reference block stride (glide/grid.py:182-188)
constexpr int REF_WIN = 16;      // reference block (active cells + 1 ring)

// Everything a cell patch needs from outside its 5 unknowns.
template <typename T> struct Patch {
    T eta[3][3];                 // eta at (i-1..i+1, j-1..j+1)
    T Hn[3][3];                  // H at the same cells ([1][1] unused: iterated)
    T bed_c, bed_l, bed_r, bed_t, bed_b;
    T beta_c, beta_l, beta_r, beta_t, beta_b;
    T g_l, g_r, g_t, g_b;        // grounded fractions of the 4 neighbours (frozen)
    T u_ll, u_rr, u_tl, u_tr, u_bl, u_br;
    T v_lt, v_lb, v_rt, v_rb, v_tt, v_bb;
    int i, j;
};

// Fill the eta window of a VYxVX tile (+ ring) and the frozen patch of the
// calling thread's cell.
template <int VY, bool CHAIN, typename T, typename P>
__device__ __forceinline__ void eta_window(T (*s_eta)[VX + 2], const T* u, const T* v, const T* B, int i0, int j0,
                                           int ny, int nx, const P& p) {
    for (int k = threadIdx.x; k < (VY + 2) * (VX + 2); k += VX * VY) {
        int r = k / (VX + 2), c = k - r * (VX + 2);
        int ic = clampi(i0 - 1 + r, 0, ny - 1), jc = clampi(j0 - 1 + c, 0, nx - 1);
        EtaIn<T> e = eta_inputs<CHAIN>(u, v, ic, jc, ny, nx);
        s_eta[r][c] = cell_eta(e, ldc<CHAIN>(B, ic, jc, ny, nx), ic, jc, ny, nx, p).eta;
    }
}

template <bool CHAIN, typename T>
__device__ __forceinline__ void load_patch(Patch<T>& P, T (*s_eta)[VX + 2], int r, int c, const T* u, const T* v,
                                           const T* H, const T* bed, const T* beta, int i, int j, int ny, int nx,
                                           const Phys<T>& p) {
    P.i = i;
    P.j = j;
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int b = 0; b < 3; b++) {
            P.eta[a][b] = s_eta[r + a][c + b];
            P.Hn[a][b] = ldc<CHAIN>(H, i - 1 + a, j - 1 + b, ny, nx);
        }
    P.bed_c = ldc<CHAIN>(bed, i, j, ny, nx); P.bed_l = ldc<CHAIN>(bed, i, j - 1, ny, nx); P.bed_r = ldc<CHAIN>(bed, i, j + 1, ny, nx);
    P.bed_t = ldc<CHAIN>(bed, i - 1, j, ny, nx); P.bed_b = ldc<CHAIN>(bed, i + 1, j, ny, nx);
    P.beta_c = ldc<CHAIN>(beta, i, j, ny, nx); P.beta_l = ldc<CHAIN>(beta, i, j - 1, ny, nx); P.beta_r = ldc<CHAIN>(beta, i, j + 1, ny, nx);
    P.beta_t = ldc<CHAIN>(beta, i - 1, j, ny, nx); P.beta_b = ldc<CHAIN>(beta, i + 1, j, ny, nx);
    P.g_l = sigmoid(P.bed_l + rho_ratio<T>() * P.Hn[1][0], p.sig_c);
    P.g_r = sigmoid(P.bed_r + rho_ratio<T>() * P.Hn[1][2], p.sig_c);
    P.g_t = sigmoid(P.bed_t + rho_ratio<T>() * P.Hn[0][1], p.sig_c);
    P.g_b = sigmoid(P.bed_b + rho_ratio<T>() * P.Hn[2][1], p.sig_c);
    P.u_ll = ldu<CHAIN>(u, i, j - 1, ny, nx); P.u_rr = ldu<CHAIN>(u, i, j + 2, ny, nx);
    P.u_tl = ldu<CHAIN>(u, i - 1, j, ny, nx); P.u_tr = ldu<CHAIN>(u, i - 1, j + 1, ny, nx);
    P.u_bl = ldu<CHAIN>(u, i + 1, j, ny, nx); P.u_br = ldu<CHAIN>(u, i + 1, j + 1, ny, nx);
    P.v_lt = ldv<CHAIN>(v, i, j - 1, ny, nx); P.v_lb = ldv<CHAIN>(v, i + 1, j - 1, ny, nx);
    P.v_rt = ldv<CHAIN>(v, i, j + 1, ny, nx); P.v_rb = ldv<CHAIN>(v, i + 1, j + 1, ny, nx);
    P.v_tt = ldv<CHAIN>(v, i - 1, j, ny, nx); P.v_bb = ldv<CHAIN>(v, i + 2, j, ny, nx);
}

template <bool CHAIN>
__device__ __forceinline__ bool ref_tile_on(const int* flags, int i, int j, int nx) {
    const int nbx = nx / REF_STRIDE + 1;
    return ld<CHAIN>(flags + (i / REF_STRIDE) * nbx + j / REF_STRIDE) != 0;
}

// Frozen per-cell coefficients of the forward local Newton loop: every term
// that depends only on neighbour values (fixed during a cell's iterations) is
// evaluated once here, so the loop only evaluates what depends on the cell's
// own 5 unknowns.  Same formulas as assemble<T,true>; the neighbour normal
// stresses are kept as k*(x - x_far) + c so no cancellation is introduced.
template <typename T> struct Frozen {
    T eta_c, ec;                       // eta of the cell, 0.25*eta
    T kl, cl, u_ll, kr, cr, u_rr;      // sxx of left/right cell
    T kt, ct, v_tt, kb, cb, v_bb;      // syy of top/bottom cell
    T S_tl, S_tr, S_bl, S_br;          // 0.25 * sum of the 3 frozen eta*H around each vertex
    T u_tl, v_lt, u_tr, v_rt, u_bl, v_lb, u_br, v_rb;
    T w_tl, w_tr, w_bl, w_br;          // vertex validity (0/1)
    T be_l, be_r, be_t, be_b;          // neighbour half of beta_eff: g*beta + (1-g)*wd
    T g_l, g_r, g_t, g_b;              // neighbour grounded fractions (gl_derivatives only)
    T beta_l, beta_r, beta_t, beta_b;
    T H_l, H_r, H_t, H_b;
    T S_l, S_r, S_t, S_b;              // neighbour surfaces max(bed,-0.917H)+H
    T db_l, db_r, db_t, db_b;          // 1 + dbase/dH of the neighbours
    T w_l, w_r, w_t, w_b;              // flux / driving validity of the 4 faces
    T bed_c, beta_c;
};

template <typename T>
__device__ __forceinline__ void make_frozen(Frozen<T>& F, const Patch<T>& P, int ny, int nx, const Phys<T>& p) {
    const int i = P.i, j = P.j;
    const T dxi = p.dxi;
    const T (&eta)[3][3] = P.eta;
    const T (&Hn)[3][3] = P.Hn;
    F.eta_c = eta[1][1];
    F.ec = T(0.25) * eta[1][1];
    T wl = (j - 1 >= 0) ? T(1) : T(0), wr = (j + 1 < nx) ? T(1) : T(0);
    T wt = (i - 1 >= 0) ? T(1) : T(0), wb = (i + 1 < ny) ? T(1) : T(0);
    T eHl = eta[1][0] * Hn[1][0], eHr = eta[1][2] * Hn[1][2], eHt = eta[0][1] * Hn[0][1], eHb = eta[2][1] * Hn[2][1];
    F.kl = T(4) * eHl * dxi * wl;  F.cl = T(2) * eHl * dxi * wl * (P.v_lt - P.v_lb);  F.u_ll = P.u_ll;
    F.kr = T(4) * eHr * dxi * wr;  F.cr = T(2) * eHr * dxi * wr * (P.v_rt - P.v_rb);  F.u_rr = P.u_rr;
    F.kt = T(4) * eHt * dxi * wt;  F.ct = T(2) * eHt * dxi * wt * (P.u_tr - P.u_tl);  F.v_tt = P.v_tt;
    F.kb = T(4) * eHb * dxi * wb;  F.cb = T(2) * eHb * dxi * wb * (P.u_br - P.u_bl);  F.v_bb = P.v_bb;
    F.S_tl = T(0.25) * (eta[0][0] * Hn[0][0] + eHt + eHl);
    F.S_tr = T(0.25) * (eHt + eta[0][2] * Hn[0][2] + eHr);
    F.S_bl = T(0.25) * (eHl + eta[2][0] * Hn[2][0] + eHb);
    F.S_br = T(0.25) * (eHr + eHb + eta[2][2] * Hn[2][2]);
    F.u_tl = P.u_tl; F.v_lt = P.v_lt; F.u_tr = P.u_tr; F.v_rt = P.v_rt;
    F.u_bl = P.u_bl; F.v_lb = P.v_lb; F.u_br = P.u_br; F.v_rb = P.v_rb;
    F.w_tl = (i > 0 && j > 0) ? T(1) : T(0);
    F.w_tr = (i > 0 && j + 1 < nx) ? T(1) : T(0);
    F.w_bl = (i + 1 < ny && j > 0) ? T(1) : T(0);
    F.w_br = (i + 1 < ny && j + 1 < nx) ? T(1) : T(0);
    F.g_l = P.g_l; F.g_r = P.g_r; F.g_t = P.g_t; F.g_b = P.g_b;
    F.beta_l = P.beta_l; F.beta_r = P.beta_r; F.beta_t = P.beta_t; F.beta_b = P.beta_b;
    F.be_l = P.g_l * P.beta_l + (T(1) - P.g_l) * p.water_drag;
    F.be_r = P.g_r * P.beta_r + (T(1) - P.g_r) * p.water_drag;
    F.be_t = P.g_t * P.beta_t + (T(1) - P.g_t) * p.water_drag;
    F.be_b = P.g_b * P.beta_b + (T(1) - P.g_b) * p.water_drag;
    F.H_l = Hn[1][0]; F.H_r = Hn[1][2]; F.H_t = Hn[0][1]; F.H_b = Hn[2][1];
    auto surf = [&](T bed, T H, T& S, T& db) {
        S = M<T>::max(bed, -rho_ratio<T>() * H) + H;
        db = T(1) + (bed > -rho_ratio<T>() * H ? T(0) : -rho_ratio<T>());
    };
    surf(P.bed_l, F.H_l, F.S_l, F.db_l);
    surf(P.bed_r, F.H_r, F.S_r, F.db_r);
    surf(P.bed_t, F.H_t, F.S_t, F.db_t);
    surf(P.bed_b, F.H_b, F.S_b, F.db_b);
    F.w_l = (j > 0 && j < nx) ? T(1) : T(0);
    F.w_r = (j + 1 < nx) ? T(1) : T(0);
    F.w_t = (i > 0 && i < ny) ? T(1) : T(0);
    F.w_b = (i + 1 < ny) ? T(1) : T(0);
    F.bed_c = P.bed_c;
    F.beta_c = P.beta_c;
}

// One local Newton step's matrix and residual from the frozen coefficients
// (same terms and order of rows/columns as assemble<T,true>).
template <typename T>
__device__ __forceinline__ void assemble_fast(const Frozen<T>& F, T ul, T ur, T vt, T vb, T Hc, T fu_l, T fu_r,
                                              T fv_t, T fv_b, T fH, T thk, T dti, const Phys<T>& p, T (&J)[25],
                                              T (&r)[5]) {
    const T dxi = p.dxi;
    const T gc = sigmoid(F.bed_c + rho_ratio<T>() * Hc, p.sig_c);
    // mass row
    {
        Calving<T> cv = calving_g(Hc, gc, p);
        Flux<T> ql = upwind_flux(ul, F.H_l, Hc, F.w_l > T(0));
        Flux<T> qr = upwind_flux(ur, Hc, F.H_r, F.w_r > T(0));
        Flux<T> qt = upwind_flux(vt, Hc, F.H_t, F.w_t > T(0));
        Flux<T> qb = upwind_flux(vb, F.H_b, Hc, F.w_b > T(0));
        T r4 = Hc * dti - fH - cv.res - ql.res * dxi + qr.res * dxi + qt.res * dxi - qb.res * dxi;
        if ((Hc - p.dt * r4) <= thk) {
            J[20] = T(0); J[21] = T(0); J[22] = T(0); J[23] = T(0); J[24] = T(1);
            r[4] = Hc - thk;
        } else {
            J[20] = -ql.d_vel * dxi;
            J[21] = qr.d_vel * dxi;
            J[22] = qt.d_vel * dxi;
            J[23] = -qb.d_vel * dxi;
            J[24] = dti - cv.d_H + (-ql.d_Hb + qr.d_Ha + qt.d_Ha - qb.d_Hb) * dxi;
            r[4] = r4;
        }
    }
    // own-cell normal stresses
    const T etaH = F.eta_c * Hc;
    const T pre = T(2) * etaH * dxi;
    const T exx = T(2) * (ur - ul) * dxi + (vt - vb) * dxi;
    const T eyy = (ur - ul) * dxi + T(2) * (vt - vb) * dxi;
    const T sxx = T(2) * etaH * exx, syy = T(2) * etaH * eyy;
    const T hx = T(2) * exx * F.eta_c * dxi, hy = T(2) * eyy * F.eta_c * dxi;
    const T p2 = pre * dxi;
    J[0] = -T(2) * p2; J[1] = T(2) * p2; J[2] = p2; J[3] = -p2; J[4] = hx;
    J[5] = T(2) * p2; J[6] = -T(2) * p2; J[7] = -p2; J[8] = p2; J[9] = -hx;
    J[10] = p2; J[11] = -p2; J[12] = -T(2) * p2; J[13] = T(2) * p2; J[14] = -hy;
    J[15] = -p2; J[16] = p2; J[17] = T(2) * p2; J[18] = -T(2) * p2; J[19] = hy;
    T r0 = -fu_l + sxx * dxi, r1 = -fu_r - sxx * dxi, r2 = -fv_t - syy * dxi, r3 = -fv_b + syy * dxi;
    // neighbour normal stresses
    r0 -= (F.kl * (ul - F.u_ll) + F.cl) * dxi;   J[0] -= F.kl * dxi;
    r1 += (F.kr * (F.u_rr - ur) + F.cr) * dxi;   J[6] -= F.kr * dxi;
    r2 += (F.kt * (F.v_tt - vt) + F.ct) * dxi;   J[12] -= F.kt * dxi;
    r3 -= (F.kb * (vb - F.v_bb) + F.cb) * dxi;   J[18] -= F.kb * dxi;
    // corner shear stresses
    {
        const T ecH = F.ec * Hc;
        T eH = (F.S_tl + ecH) * F.w_tl;
        T exy = T(0.5) * ((F.u_tl - ul) * dxi + (vt - F.v_lt) * dxi);
        T res = T(2) * eH * exy * dxi, dd = eH * dxi * dxi, de = T(2) * exy * F.w_tl * F.ec * dxi;
        r0 += res; r2 -= res; J[0] -= dd; J[4] += de; J[12] -= dd; J[14] -= de;
        eH = (F.S_tr + ecH) * F.w_tr;
        exy = T(0.5) * ((F.u_tr - ur) * dxi + (F.v_rt - vt) * dxi);
        res = T(2) * eH * exy * dxi; dd = eH * dxi * dxi; de = T(2) * exy * F.w_tr * F.ec * dxi;
        r1 += res; r2 += res; J[6] -= dd; J[9] += de; J[12] -= dd; J[14] += de;
        eH = (F.S_bl + ecH) * F.w_bl;
        exy = T(0.5) * ((ul - F.u_bl) * dxi + (vb - F.v_lb) * dxi);
        res = T(2) * eH * exy * dxi; dd = eH * dxi * dxi; de = T(2) * exy * F.w_bl * F.ec * dxi;
        r0 -= res; r3 -= res; J[0] -= dd; J[4] -= de; J[18] -= dd; J[19] -= de;
        eH = (F.S_br + ecH) * F.w_br;
        exy = T(0.5) * ((ur - F.u_br) * dxi + (F.v_rb - vb) * dxi);
        res = T(2) * eH * exy * dxi; dd = eH * dxi * dxi; de = T(2) * exy * F.w_br * F.ec * dxi;
        r1 -= res; r3 += res; J[6] -= dd; J[9] -= de; J[18] -= dd; J[19] += de;
    }
    // basal drag
    {
        const T bec = gc * F.beta_c + (T(1) - gc) * p.water_drag;
        T bl = T(0.5) * (F.be_l + bec), br = T(0.5) * (bec + F.be_r);
        T bt = T(0.5) * (F.be_t + bec), bb = T(0.5) * (bec + F.be_b);
        r0 -= bl * ul; r1 -= br * ur; r2 -= bt * vt; r3 -= bb * vb;
        J[0] -= bl; J[6] -= br; J[12] -= bt; J[18] -= bb;
        if (p.gl_deriv) {
            T dgc = rho_ratio<T>() * (p.sig_c * gc * (T(1) - gc)) * (F.beta_c - p.water_drag);
            J[4] += T(-0.5) * dgc * ul;
            J[9] += T(-0.5) * dgc * ur;
            J[14] += T(-0.5) * dgc * vt;
            J[19] += T(-0.5) * dgc * vb;
        }
    }
    // driving stress; x: left (m) / right (p); y: bottom (m) / top (p)
    {
        const T bc = M<T>::max(F.bed_c, -rho_ratio<T>() * Hc);
        const T Sc = bc + Hc;
        const T dbc = T(1) + (F.bed_c > -rho_ratio<T>() * Hc ? T(0) : -rho_ratio<T>());
        // left face: m = left, p = this cell
        T Havg = T(0.5) * (F.H_l + Hc), dS = Sc - F.S_l;
        r0 -= Havg * dS * dxi * F.w_l;
        J[4] -= (T(0.5) * dS * dxi + Havg * dbc * dxi) * F.w_l;
        // right face: m = this cell, p = right
        Havg = T(0.5) * (Hc + F.H_r); dS = F.S_r - Sc;
        r1 -= Havg * dS * dxi * F.w_r;
        J[9] -= (T(0.5) * dS * dxi - Havg * dbc * dxi) * F.w_r;
        // top face: m = this cell (bottom), p = top
        Havg = T(0.5) * (Hc + F.H_t); dS = F.S_t - Sc;
        r2 -= Havg * dS * dxi * F.w_t;
        J[14] -= (T(0.5) * dS * dxi - Havg * dbc * dxi) * F.w_t;
        // bottom face: m = bottom, p = this cell (top)
        Havg = T(0.5) * (F.H_b + Hc); dS = Sc - F.S_b;
        r3 -= Havg * dS * dxi * F.w_b;
        J[19] -= (T(0.5) * dS * dxi + Havg * dbc * dxi) * F.w_b;
    }
    r[0] = r0; r[1] = r1; r[2] = r2; r[3] = r3;
}

// LU solve with the pivot reciprocals reused in the back substitution.
template <typename T> __device__ __forceinline__ void lu5_solve_fast(T (&A)[25], const T (&b)[5], T (&x)[5]) {
    T inv[5];
#pragma unroll
    for (int k = 0; k < 5; k++) {
        inv[k] = M<T>::rcp(A[k * 5 + k]);
#pragma unroll
        for (int i = k + 1; i < 5; i++) {
            A[i * 5 + k] *= inv[k];
#pragma unroll
            for (int j = k + 1; j < 5; j++) A[i * 5 + j] -= A[i * 5 + k] * A[k * 5 + j];
        }
    }
    T y1 = b[1] - A[5] * b[0];
    T y2 = b[2] - A[10] * b[0] - A[11] * y1;
    T y3 = b[3] - A[15] * b[0] - A[16] * y1 - A[17] * y2;
    T y4 = b[4] - A[20] * b[0] - A[21] * y1 - A[22] * y2 - A[23] * y3;
    x[4] = y4 * inv[4];
    x[3] = (y3 - A[19] * x[4]) * inv[3];
    x[2] = (y2 - A[13] * x[3] - A[14] * x[4]) * inv[2];
    x[1] = (y1 - A[7] * x[2] - A[8] * x[3] - A[9] * x[4]) * inv[1];
    x[0] = (b[0] - A[1] * x[1] - A[2] * x[2] - A[3] * x[3] - A[4] * x[4]) * inv[0];
}

// 5x5 solve with partial (row) pivoting, the robustness variant of the
// reference (lu_5x5_solve_pivot, glide/cuda/common.cu:180-233): the largest
// |entry| of the column becomes the pivot (first one on ties), a pivot below
// 1e-14 in magnitude skips its elimination step, a diagonal below 1e-14 in
// back substitution gives x = 0.  Rows are swapped in registers by unrolled
// conditional moves.
template <typename T> __device__ __forceinline__ void lu5_solve_pivot(T (&A)[25], const T (&b)[5], T (&x)[5]) {
    T y[5] = {b[0], b[1], b[2], b[3], b[4]};
    const T tiny = T(1e-14);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        int p = k;
        T best = M<T>::abs(A[k * 5 + k]);
#pragma unroll
        for (int i = k + 1; i < 5; i++) {
            const T a = M<T>::abs(A[i * 5 + k]);
            if (a > best) {
                best = a;
                p = i;
            }
        }
#pragma unroll
        for (int i = k + 1; i < 5; i++) {
            if (i == p) {
#pragma unroll
                for (int j = 0; j < 5; j++) {
                    const T t = A[k * 5 + j];
                    A[k * 5 + j] = A[i * 5 + j];
                    A[i * 5 + j] = t;
                }
                const T t = y[k];
                y[k] = y[i];
                y[i] = t;
            }
        }
        const T piv = A[k * 5 + k];
        if (M<T>::abs(piv) < tiny) continue;
#pragma unroll
        for (int i = k + 1; i < 5; i++) {
            const T f = A[i * 5 + k] / piv;
            A[i * 5 + k] = f;
#pragma unroll
            for (int j = k + 1; j < 5; j++) A[i * 5 + j] -= f * A[k * 5 + j];
        }
    }
#pragma unroll
    for (int i = 1; i < 5; i++) {
#pragma unroll
        for (int j = 0; j < i; j++) y[i] -= A[i * 5 + j] * y[j];
    }
#pragma unroll
    for (int i = 4; i >= 0; i--) {
        T v = y[i];
#pragma unroll
        for (int j = i + 1; j < 5; j++) v -= A[i * 5 + j] * x[j];
        const T d = A[i * 5 + i];
        x[i] = M<T>::abs(d) > tiny ? v / d : T(0);
    }
}

// Per-cell Newton deltas.  scratch holds 5 cell arrays: 0.5*du_l, 0.5*du_r,
// 0.5*dv_t, 0.5*dv_b, dH.
template <typename T, int VY, bool LOCAL, bool CHAIN, typename P>
#ifndef GLIDE_VANKA64_MIN_BLOCKS
#define GLIDE_VANKA64_MIN_BLOCKS 2
#endif
#ifndef GLIDE_VANKA32_MIN_BLOCKS
#define GLIDE_VANKA32_MIN_BLOCKS 2
#endif
__global__ void __launch_bounds__(VX * VY, (sizeof(T) == 4 ? GLIDE_VANKA32_MIN_BLOCKS : GLIDE_VANKA64_MIN_BLOCKS) * (8 / VY)) vanka_cells_kernel(
    T* __restrict__ scratch, const T* __restrict__ u, const T* __restrict__ v, const T* __restrict__ H,
    const T* __restrict__ f_u, const T* __restrict__ f_v, const T* __restrict__ f_H, const T* __restrict__ bed,
    const T* __restrict__ B, const T* __restrict__ beta, const T* __restrict__ gamma, const int* __restrict__ flags,
    const int* __restrict__ any_active, int n_newton, T shift, T step, int pivot, Geo g, P p) {
    __shared__ T s_eta[VY + 2][VX + 2];
    const int zero = chain_enter<CHAIN>();
    const int ny = g.ny, nx = g.nx;
    const int bz = blockIdx.z + zero;
    if (LOCAL && ld<CHAIN>(any_active + bz) == 0) return;
    u += bz * g.nu(); v += bz * g.nv(); H += bz * g.nc(); f_u += bz * g.nu(); f_v += bz * g.nv();
    f_H += bz * g.nc(); bed += bz * g.nc(); B += bz * g.nc(); beta += bz * g.nc(); gamma += bz * g.nc();
    const int64_t nc = g.nc();
    scratch += bz * 5 * nc;
    if (LOCAL) flags += bz * int64_t(ny / REF_STRIDE + 1) * (nx / REF_STRIDE + 1);
    const int i0 = blockIdx.y * VY + zero, j0 = blockIdx.x * VX;
    const int r = threadIdx.x / VX, c = threadIdx.x % VX;
    const int i = i0 + r, j = j0 + c;
    eta_window<VY, CHAIN>(s_eta, u, v, B, i0, j0, ny, nx, p);
    __syncthreads();
    if (i >= ny || j >= nx) return;
    if (LOCAL && !ref_tile_on<CHAIN>(flags, i, j, nx)) return;

    Frozen<T> F;
    {
        Patch<T> pt;
        load_patch<CHAIN>(pt, s_eta, r, c, u, v, H, bed, beta, i, j, ny, nx, p);
        make_frozen<T>(F, pt, ny, nx, p);
    }
    // 32-bit offsets within one field (the entry points bound a field below 2^31 elements)
    const int iu = i * (nx + 1) + j, ic32 = i * nx + j;
    const T ul0 = ld<CHAIN>(u + iu), ur0 = ld<CHAIN>(u + iu + 1);
    const T vt0 = ld<CHAIN>(v + ic32), vb0 = ld<CHAIN>(v + ic32 + nx);
    const T H0 = ld<CHAIN>(H + ic32);
    const T fu_l = ld<CHAIN>(f_u + iu), fu_r = ld<CHAIN>(f_u + iu + 1);
    const T fv_t = ld<CHAIN>(f_v + ic32), fv_b = ld<CHAIN>(f_v + ic32 + nx);
    const T fH = ld<CHAIN>(f_H + ic32);
    const T thk = ld<CHAIN>(gamma + ic32);
    const T dti = T(1) / p.dt;
    T ul = ul0, ur = ur0, vt = vt0, vb = vb0, Hc = H0;
    for (int it = 0; it < n_newton; it++) {
        T J[25], rr[5], x[5];
        assemble_fast<T>(F, ul, ur, vt, vb, Hc, fu_l, fu_r, fv_t, fv_b, fH, thk, dti, p, J, rr);
        J[0] -= shift; J[6] -= shift; J[12] -= shift; J[18] -= shift; J[24] += shift;  // vanka.cu:406-410
        if (sizeof(T) == 8 || pivot)   // FP64 comes here for pivoted solves only
            lu5_solve_pivot(J, rr, x);
        else
            lu5_solve_fast(J, rr, x);
        ul -= step * x[0];  // reference step 0.25: relaxation_factor, glide/cuda/vanka.cu:416
        ur -= step * x[1];
        vt -= step * x[2];
        vb -= step * x[3];
        Hc -= step * x[4];
        Hc = M<T>::max(Hc, thk);
    }
    if (!(isfinite(ul) && isfinite(ur) && isfinite(vt) && isfinite(vb) && isfinite(Hc))) {
        ul = ul0, ur = ur0, vt = vt0, vb = vb0, Hc = H0;  // a failed local solve leaves its cell unchanged
    }
    const int64_t ic = int64_t(i) * nx + j;
    scratch[ic] = T(0.5) * (ul - ul0);
    scratch[nc + ic] = T(0.5) * (ur - ur0);
    scratch[2 * nc + ic] = T(0.5) * (vt - vt0);
    scratch[3 * nc + ic] = T(0.5) * (vb - vb0);
    scratch[4 * nc + ic] = Hc - H0;
}

// U += omega * delta, face delta = sum of the two adjacent cells' halves.
template <typename T, bool LOCAL, bool CHAIN>
__global__ void vanka_apply_kernel(T* __restrict__ u, T* __restrict__ v, T* __restrict__ H,
                                   const T* __restrict__ scratch, const int* __restrict__ flags,
                                   const int* __restrict__ any_active, T omega, Geo g) {
    const int zero = chain_enter<CHAIN>();
    const int ny = g.ny, nx = g.nx;
    const int bz = blockIdx.z + zero;
    if (LOCAL && ld<CHAIN>(any_active + bz) == 0) return;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y * blockDim.y + threadIdx.y + zero;
    if (i > ny || j > nx) return;
    const int64_t nc = g.nc();
    u += bz * g.nu(); v += bz * g.nv(); H += bz * g.nc();
    scratch += bz * 5 * nc;
    if (LOCAL) flags += bz * int64_t(ny / REF_STRIDE + 1) * (nx / REF_STRIDE + 1);
    auto on = [&](int ii, int jj) { return !LOCAL || ref_tile_on<CHAIN>(flags, ii, jj, nx); };
    if (i < ny) {  // u-face (i,j), j in [0,nx]
        T d = T(0);
        if (j < nx && on(i, j)) d += ld<CHAIN>(scratch + int64_t(i) * nx + j);                   // as u_l of cell (i,j)
        if (j > 0 && on(i, j - 1)) d += ld<CHAIN>(scratch + nc + int64_t(i) * nx + j - 1);        // as u_r of cell (i,j-1)
        u[int64_t(i) * (nx + 1) + j] += omega * d;
    }
    if (j < nx) {  // v-face (i,j), i in [0,ny]
        T d = T(0);
        if (i < ny && on(i, j)) d += ld<CHAIN>(scratch + 2 * nc + int64_t(i) * nx + j);
        if (i > 0 && on(i - 1, j)) d += ld<CHAIN>(scratch + 3 * nc + int64_t(i - 1) * nx + j);
        v[int64_t(i) * nx + j] += omega * d;
    }
    if (i < ny && j < nx && on(i, j)) H[int64_t(i) * nx + j] += omega * ld<CHAIN>(scratch + 4 * nc + int64_t(i) * nx + j);
}

// Local error indicator (glide/solver.py:148-154) and reference-tile flags.
// err = |r_u(l)| + |r_u(r)| + |r_v(t)| + |r_v(b)| + |FB(r_H, H-gamma)| > threshold
template <typename T>
__global__ void error_mask_kernel(T* __restrict__ err_mask, const T* __restrict__ r_u, const T* __restrict__ r_v,
                                  const T* __restrict__ r_H, const T* __restrict__ H, const T* __restrict__ gamma,
                                  T threshold, Geo g) {
    const int zero = chain_enter<true>();
    const int ny = g.ny, nx = g.nx;
    const int bz = blockIdx.z + zero;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y * blockDim.y + threadIdx.y + zero;
    if (i >= ny || j >= nx) return;
    r_u += bz * g.nu(); r_v += bz * g.nv(); r_H += bz * g.nc(); H += bz * g.nc(); gamma += bz * g.nc();
    err_mask += bz * g.nc();
    const int64_t ic = int64_t(i) * nx + j;
    T a = ld<true>(r_H + ic), b = ld<true>(H + ic) - ld<true>(gamma + ic);
    T fb = a + b - M<T>::sqrt(a * a + b * b);
    T tot = M<T>::abs(ld<true>(r_u + int64_t(i) * (nx + 1) + j + 1)) +
            M<T>::abs(ld<true>(r_u + int64_t(i) * (nx + 1) + j)) + M<T>::abs(ld<true>(r_v + int64_t(i + 1) * nx + j)) +
            M<T>::abs(ld<true>(r_v + ic)) + M<T>::abs(fb);
    err_mask[ic] = tot > threshold ? T(1) : T(0);
}

// One CTA per reference block: flag = any in-domain cell of the 16x16 window
// has err_mask > 0.5.  any_active[b] counts active blocks.
template <typename T>
__global__ void tile_flags_kernel(int* __restrict__ flags, int* __restrict__ any_active,
                                  const T* __restrict__ err_mask, Geo g) {
    const int ny = g.ny, nx = g.nx;
    const int bz = blockIdx.z;
    const int nbx = nx / REF_STRIDE + 1;
    const int bx = blockIdx.x, by = blockIdx.y;
    err_mask += bz * g.nc();
    flags += bz * int64_t(ny / REF_STRIDE + 1) * nbx;
    const int i = by * REF_STRIDE - 1 + threadIdx.y;
    const int j = bx * REF_STRIDE - 1 + threadIdx.x;
    bool bad = (i >= 0 && i < ny && j >= 0 && j < nx) && err_mask[int64_t(i) * nx + j] > T(0.5);
    int any = __syncthreads_or(bad);
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        flags[by * nbx + bx] = any;
        if (any) atomicAdd(any_active + bz, 1);
    }
}

// --------------------------------------------------------------------------
// launchers
// --------------------------------------------------------------------------
static inline dim3 cell_grid(const Geo& g, int vy) { return dim3((g.nx + VX - 1) / VX, (g.ny + vy - 1) / vy, g.nb); }
static inline dim3 face_grid(const Geo& g) { return dim3((g.nx + 1 + 31) / 32, (g.ny + 1 + 7) / 8, g.nb); }

// Tile height.  A cell's Newton loop is one long dependent chain, so on a grid
// that leaves SMs idle a warp should share its scheduler with as few others as
// possible: quarter-SM tiles of 4 rows up to 32 tiles of 8 (64^2), and up to 96
// (128^2) single-row tiles of one warp, which the block scheduler spreads
// evenly.  Microseconds per sweep of 10 Newton steps, FP32, 8 / 4 / 1 rows:
// 32^2 10.3 / 8.3 / 8.7, 64^2 10.5 / 8.6 / 9.4, 128^2 11.6 / 12.7 / 9.5, 256^2
// 15.8 / 16.6 / 17.8.
static inline int cell_tile(const Geo& g) {
    const int64_t tiles = blocks_of(cell_grid(g, 8));
    return tiles <= 32 ? 4 : tiles <= 96 ? 1 : 8;
}
// Which form of the cell kernel: the march (vanka_march.cu) in FP64, and in
// FP32 for sweeps of their own from 2^16 cells on.  The FP32 FAS cycle keeps
// the tile form at every size although the march is faster there too (512^2:
// 47 us per sweep of 10 Newton steps against 38): the two round differently, and
// a few FP32 cycles amplify a rounding 1e3 to 1e4 times, so a step's answer
// would move by up to 3e-4 between the forms.  Pivoted local solves exist in the
// tile form only.  Microseconds per sweep, tile / march: FP32 of 10 steps 256^2
// 16.1 / 13.3, 1024^2 174 / 136, of 2 steps 1024^2 73.5 / 50.3; 64^2 and below
// within 10 % of each other; FP64 of 10 steps 32^2 16.5 / 13.3, 256^2 33.9 /
// 26.2, 1024^2 408 / 348, of 2 steps 32^2 7.7 / 8.1, 1024^2 168 / 141.
template <typename T> static inline bool use_march(const Geo& g, int pivot, bool cycle) {
    if (pivot) return false;
    return sizeof(T) == 8 || (!cycle && g.nc() * g.nb >= (int64_t(1) << 16));
}
// The sweep's two kernels are chained while they fit the chip about once; not
// with single-row tiles, whose CTAs would be placed around those of the kernel
// before and lose their even spread (128^2: 12.9 us per sweep chained, 9.5 not).
static inline bool sweep_chained(const Geo& g, bool march) {
    return (march || cell_tile(g) != 1) && blocks_of(cell_grid(g, 8)) <= 592;
}
template <typename T>
void run_march(const GlideLevelArgs*, const void*, const void*, const void*, int, double, double, const int*,
               const int*, void*, cudaStream_t);

template <typename T>
static void run_cells(const GlideLevelArgs* a, const void* f_u, const void* f_v, const void* f_H, int n_newton,
                      double shift, double step, int pivot, const int* flags, const int* any_active, void* scratch,
                      const Geo& g, bool cycle, cudaStream_t s) {
    if (use_march<T>(g, pivot, cycle)) {
        run_march<T>(a, f_u, f_v, f_H, n_newton, shift, step, flags, any_active, scratch, s);
        return;
    }
    with_glen(a->params, make_phys<T>(a->params, a->dx, a->dt), [&](auto p) {
        using P = decltype(p);
        auto go = [&](auto vy, auto chain) {
            constexpr int VY = decltype(vy)::value;
            constexpr bool CHAIN = decltype(chain)::value;
            auto run = [&](auto kernel) {
                launch_chained<CHAIN>(kernel, cell_grid(g, VY), VX * VY, s, (T*)scratch, (const T*)a->u,
                                      (const T*)a->v, (const T*)a->H, (const T*)f_u, (const T*)f_v, (const T*)f_H,
                                      (const T*)a->bed, (const T*)a->B, (const T*)a->beta, (const T*)a->gamma, flags,
                                      any_active, n_newton, T(shift), T(step), pivot, g, p);
            };
            flags ? run(vanka_cells_kernel<T, VY, true, CHAIN, P>) : run(vanka_cells_kernel<T, VY, false, CHAIN, P>);
        };
        using std::integral_constant;
        const int vy = cell_tile(g);
        if (vy == 4)
            go(integral_constant<int, 4>{}, std::true_type{});
        else if (vy == 1)
            go(integral_constant<int, 1>{}, std::false_type{});
        else if (sweep_chained(g, false))
            go(integral_constant<int, 8>{}, std::true_type{});
        else
            go(integral_constant<int, 8>{}, std::false_type{});
    });
}

template <typename T>
int launch_vanka_sweeps(const GlideLevelArgs* a, const void* f_u, const void* f_v, const void* f_H, int n_iter,
                        int n_newton, double omega, double shift, const int* flags, const int* any_active,
                        void* scratch, cudaStream_t s, double newton_step, int pivot, bool cycle) {
    Geo g{a->ny, a->nx, a->nb};
    auto apply = [&](auto chain) {
        constexpr bool CHAIN = decltype(chain)::value;
        auto run = [&](auto kernel) {
            launch_chained<CHAIN>(kernel, face_grid(g), dim3(32, 8), s, (T*)a->u, (T*)a->v, (T*)a->H,
                                  (const T*)scratch, flags, any_active, T(omega), g);
        };
        flags ? run(vanka_apply_kernel<T, true, CHAIN>) : run(vanka_apply_kernel<T, false, CHAIN>);
    };
    const bool chained = sweep_chained(g, use_march<T>(g, pivot, cycle));
    for (int k = 0; k < n_iter; k++) {
        run_cells<T>(a, f_u, f_v, f_H, n_newton, shift, newton_step, pivot, flags, any_active, scratch, g, cycle, s);
        chained ? apply(std::true_type{}) : apply(std::false_type{});
    }
    return (int)cudaGetLastError();
}

// Only the per-cell Newton kernel, n_launch times (profiling / timing; U is not updated).
template <typename T>
int launch_vanka_cells(const GlideLevelArgs* a, const void* f_u, const void* f_v, const void* f_H, int n_launch,
                       int n_newton, double shift, const int* flags, const int* any_active, void* scratch,
                       cudaStream_t s, double newton_step) {
    Geo g{a->ny, a->nx, a->nb};
    for (int k = 0; k < n_launch; k++)
        run_cells<T>(a, f_u, f_v, f_H, n_newton, shift, newton_step, 0, flags, any_active, scratch, g, false, s);
    return (int)cudaGetLastError();
}

template <typename T>
int launch_error_mask(const GlideLevelArgs* a, const void* r_u, const void* r_v, const void* r_H, double threshold,
                      void* err_mask, int* flags, int* any_active, cudaStream_t s) {
    Geo g{a->ny, a->nx, a->nb};
    dim3 blk(32, 8);
    dim3 grd((g.nx + 31) / 32, (g.ny + 7) / 8, g.nb);
    launch_chained<true>(error_mask_kernel<T>, grd, blk, s, (T*)err_mask, (const T*)r_u, (const T*)r_v, (const T*)r_H,
                                             (const T*)a->H, (const T*)a->gamma, T(threshold), g);
    if (flags) {
        cudaMemsetAsync(any_active, 0, sizeof(int) * g.nb, s);
        dim3 tg(g.nx / REF_STRIDE + 1, g.ny / REF_STRIDE + 1, g.nb);
        glide::count_launch(), tile_flags_kernel<T><<<tg, dim3(REF_WIN, REF_WIN), 0, s>>>(flags, any_active, (const T*)err_mask, g);
    }
    return (int)cudaGetLastError();
}

template <typename T>
int launch_tile_flags(const GlideLevelArgs* a, const void* err_mask, int* flags, int* any_active, cudaStream_t s) {
    Geo g{a->ny, a->nx, a->nb};
    cudaMemsetAsync(any_active, 0, sizeof(int) * g.nb, s);
    dim3 tg(g.nx / REF_STRIDE + 1, g.ny / REF_STRIDE + 1, g.nb);
    glide::count_launch(), tile_flags_kernel<T><<<tg, dim3(REF_WIN, REF_WIN), 0, s>>>(flags, any_active, (const T*)err_mask, g);
    return (int)cudaGetLastError();
}

#define INST(T)                                                                                                  \
    template int launch_vanka_sweeps<T>(const GlideLevelArgs*, const void*, const void*, const void*, int, int,   \
                                        double, double, const int*, const int*, void*, cudaStream_t, double, int, bool);\
    template int launch_vanka_cells<T>(const GlideLevelArgs*, const void*, const void*, const void*, int, int,     \
                                       double, const int*, const int*, void*, cudaStream_t, double);              \
    template int launch_error_mask<T>(const GlideLevelArgs*, const void*, const void*, const void*, double,       \
                                      void*, int*, int*, cudaStream_t);                                           \
    template int launch_tile_flags<T>(const GlideLevelArgs*, const void*, int*, int*, cudaStream_t);
INST(float)
INST(double)
#undef INST

}  // namespace glide
