// Cell-patch Vanka smoothers (glide/cuda/vanka.cu) on B200.
//
// Forward sweep:
//   the cell kernel runs the damped local Newton iterations on each cell's 5
//     unknowns (u_l, u_r, v_t, v_b, H_c) with the neighbours and the viscosity
//     frozen, and stores half of each face change and the full H change per
//     cell (deterministic, no atomics): here a thread per cell of a tile
//     (vanka_cells), in vanka_march.cu a march down rows; use_march chooses;
//   the update: every face adds the halves of its two cells, U += omega*delta
//     (the reference zero-fills a delta vector, scatters with atomicAdd and
//     axpys on the host: glide/grid.py:305-317, vanka.cu:433-437); by the next
//     sweep's cell kernel as it reads the state, or by vanka_apply.
// In the tile form the state in reach of a tile is read (and updated) once into
// shared memory and the viscosity of the tile plus a one-cell ring computed
// there; the neighbours' grounding sigmoids are hoisted out of the Newton loop.
// The local variant gates cells by the reference's 16x16-window / stride-14
// block rule (vanka.cu:875-888) through per-tile flags.
//
// What bounds the tile form: below about 200^2 the latency of one cell's chain
// (0.33 us per Newton step, 3 us to read, assemble and store), above it
// instruction issue (4,870 instructions per warp of 32 cells and 10 steps).
#include <type_traits>

#include "cell_system.cuh"

namespace glide {

// A tile is VX x VY cells, a CTA of four warps.  A cell's Newton loop is one long
// dependent chain, so on a grid that leaves SMs idle a warp should share its
// scheduler with as few others as possible, and on a large one small CTAs even
// out the last wave: tiles of 8 rows took 8.9 us per sweep of 10 Newton steps
// at 128^2 against 7.1 (FP32), 45.1 against 44.6 at 512^2, 176 against 172 at
// 1024^2 (85 against 74 of 2 steps); single rows 9.1 at 128^2.
constexpr int VX = 32, VY = 4;
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

template <bool CHAIN>
__device__ __forceinline__ bool ref_tile_on(const int* flags, int i, int j, int nx) {
    const int nbx = nx / REF_STRIDE + 1;
    return ld<CHAIN>(flags + (i / REF_STRIDE) * nbx + j / REF_STRIDE) != 0;
}

// The state a sweep starts from: U itself, or U plus the update of the sweep
// before it (has; d*: that sweep's five cell arrays).  The update is
// vanka_apply_kernel's, term by term, so both ways give the same bits.  Loads
// and sums are apart, so that a thread has all its loads in flight at once: the
// latency of this read is most of a small grid's sweep outside its Newton steps.
template <typename T, bool LOCAL, bool CHAIN> struct State {
    const T *u, *v, *H;
    const T *du_l, *du_r, *dv_t, *dv_b, *dH;   // readable (any cell array) without an update
    const int* flags;
    T omega;
    int ny, nx;
    bool has;
    struct In { T x, a, b; int fa, fb; };
    __device__ __forceinline__ void two(In& q, const T* da, int ia, int ja, const T* db, int ib, int jb) const {
        ia = min(ia, ny - 1); ja = min(ja, nx - 1); ib = max(ib, 0); jb = max(jb, 0);   // in range where unused
        q.a = ld<CHAIN>(da + (ia * nx + ja));
        q.b = ld<CHAIN>(db + (ib * nx + jb));
        if (LOCAL) {
            const int nbx = nx / REF_STRIDE + 1;
            q.fa = ld<CHAIN>(flags + (ia / REF_STRIDE) * nbx + ja / REF_STRIDE);
            q.fb = ld<CHAIN>(flags + (ib / REF_STRIDE) * nbx + jb / REF_STRIDE);
        }
    }
    __device__ __forceinline__ T sum(const In& q, bool first, bool second) const {
        T d = T(0);
        d += first && (!LOCAL || q.fa) ? q.a : T(0);
        d += second && (!LOCAL || q.fb) ? q.b : T(0);
        return has ? q.x + omega * d : q.x;
    }
    // u-face (i,j): u_l of cell (i,j), u_r of cell (i,j-1)
    __device__ __forceinline__ In loadU(int i, int j) const {
        In q;
        q.x = ld<CHAIN>(u + (i * (nx + 1) + j));
        two(q, du_l, i, j, du_r, i, j - 1);
        return q;
    }
    __device__ __forceinline__ T sumU(const In& q, int, int j) const { return sum(q, j < nx, j > 0); }
    __device__ __forceinline__ In loadV(int i, int j) const {
        In q;
        q.x = ld<CHAIN>(v + (i * nx + j));
        two(q, dv_t, i, j, dv_b, i - 1, j);
        return q;
    }
    __device__ __forceinline__ T sumV(const In& q, int i, int) const { return sum(q, i < ny, i > 0); }
    __device__ __forceinline__ In loadH(int i, int j) const {
        In q;
        q.x = ld<CHAIN>(H + (i * nx + j));
        q.a = ld<CHAIN>(dH + (i * nx + j));
        if (LOCAL) q.fa = ld<CHAIN>(flags + (i / REF_STRIDE) * (nx / REF_STRIDE + 1) + j / REF_STRIDE);
        return q;
    }
    __device__ __forceinline__ T sumH(const In& q) const {
        return has && (!LOCAL || q.fa) ? q.x + omega * q.a : q.x;
    }
};

// The state in reach of a tile's cells, clamped at the domain's edges: entry
// (r, c) of u is face (i0-2+r, j0-1+c), of v (i0-1+r, j0-2+c), of H cell
// (i0-1+r, j0-1+c).
template <typename T> struct Window {
    T u[VY + 4][VX + 3], v[VY + 3][VX + 4], H[VY + 2][VX + 2], eta[VY + 2][VX + 2];
};

// Fill the state of the window; the tile's own entries also go to (ou, ov, oH)
// unless null (faces belong to the cell right of / below them, a domain's last
// face to its last tile).
template <typename S, typename T>
__device__ __forceinline__ void state_window(Window<T>& W, const S& st, T* ou, T* ov, T* oH, int i0, int j0) {
    constexpr int NT = VX * VY, CU = VX + 3, CV = VX + 4, CH = VX + 2;
    constexpr int NU = (VY + 4) * CU, NV = (VY + 3) * CV, NH = (VY + 2) * CH;
    constexpr int KU = (NU + NT - 1) / NT, KV = (NV + NT - 1) / NT, KH = (NH + NT - 1) / NT;
    const int ny = st.ny, nx = st.nx;
    const int ie = min(i0 + VY, ny), je = min(j0 + VX, nx);
    const bool lastr = ie == ny, lastc = je == nx;
    typename S::In qu[KU], qv[KV], qh[KH];
#pragma unroll
    for (int m = 0; m < KU; m++) {
        const int k = min(int(threadIdx.x) + m * NT, NU - 1), r = k / CU, c = k - r * CU;
        qu[m] = st.loadU(clampi(i0 - 2 + r, 0, ny - 1), clampi(j0 - 1 + c, 0, nx));
    }
#pragma unroll
    for (int m = 0; m < KV; m++) {
        const int k = min(int(threadIdx.x) + m * NT, NV - 1), r = k / CV, c = k - r * CV;
        qv[m] = st.loadV(clampi(i0 - 1 + r, 0, ny), clampi(j0 - 2 + c, 0, nx - 1));
    }
#pragma unroll
    for (int m = 0; m < KH; m++) {
        const int k = min(int(threadIdx.x) + m * NT, NH - 1), r = k / CH, c = k - r * CH;
        qh[m] = st.loadH(clampi(i0 - 1 + r, 0, ny - 1), clampi(j0 - 1 + c, 0, nx - 1));
    }
#pragma unroll
    for (int m = 0; m < KU; m++) {
        const int k = min(int(threadIdx.x) + m * NT, NU - 1), r = k / CU, c = k - r * CU;
        const int i = i0 - 2 + r, j = j0 - 1 + c;
        const T x = st.sumU(qu[m], clampi(i, 0, ny - 1), clampi(j, 0, nx));
        W.u[r][c] = x;
        if (ou && i >= i0 && i < ie && j >= j0 && (j < je || (lastc && j == nx))) ou[i * (nx + 1) + j] = x;
    }
#pragma unroll
    for (int m = 0; m < KV; m++) {
        const int k = min(int(threadIdx.x) + m * NT, NV - 1), r = k / CV, c = k - r * CV;
        const int i = i0 - 1 + r, j = j0 - 2 + c;
        const T x = st.sumV(qv[m], clampi(i, 0, ny), clampi(j, 0, nx - 1));
        W.v[r][c] = x;
        if (ou && i >= i0 && (i < ie || (lastr && i == ny)) && j >= j0 && j < je) ov[i * nx + j] = x;
    }
#pragma unroll
    for (int m = 0; m < KH; m++) {
        const int k = min(int(threadIdx.x) + m * NT, NH - 1), r = k / CH, c = k - r * CH;
        const int i = i0 - 1 + r, j = j0 - 1 + c;
        const T x = st.sumH(qh[m]);
        W.H[r][c] = x;
        if (ou && i >= i0 && i < ie && j >= j0 && j < je) oH[i * nx + j] = x;
    }
}

// Fill the eta window of a VYxVX tile (+ ring).
template <bool CHAIN, typename T, typename P>
__device__ __forceinline__ void eta_window(Window<T>& W, const T* B, int i0, int j0, int ny, int nx, const P& p) {
    for (int k = threadIdx.x; k < (VY + 2) * (VX + 2); k += VX * VY) {
        int r = k / (VX + 2), c = k - r * (VX + 2);
        int ic = clampi(i0 - 1 + r, 0, ny - 1), jc = clampi(j0 - 1 + c, 0, nx - 1);
        const int a = ic - i0, b = jc - j0;
        EtaIn<T> e;
        e.ul = W.u[a + 2][b + 1];    e.ur = W.u[a + 2][b + 2];
        e.vt = W.v[a + 1][b + 2];    e.vb = W.v[a + 2][b + 2];
        e.u_tl = W.u[a + 1][b + 1];  e.u_tr = W.u[a + 1][b + 2];
        e.u_bl = W.u[a + 3][b + 1];  e.u_br = W.u[a + 3][b + 2];
        e.v_lt = W.v[a + 1][b + 1];  e.v_rt = W.v[a + 1][b + 3];
        e.v_lb = W.v[a + 2][b + 1];  e.v_rb = W.v[a + 2][b + 3];
        W.eta[r][c] = cell_eta(e, ldc<CHAIN>(B, ic, jc, ny, nx), ic, jc, ny, nx, p).eta;
    }
}

// The frozen patch of cell (r, c) of the tile.
template <bool CHAIN, typename T>
__device__ __forceinline__ void load_patch(Patch<T>& P, const Window<T>& W, int r, int c, const T* bed,
                                           const T* beta, int i, int j, int ny, int nx, const Phys<T>& p) {
    P.i = i;
    P.j = j;
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int b = 0; b < 3; b++) {
            P.eta[a][b] = W.eta[r + a][c + b];
            P.Hn[a][b] = W.H[r + a][c + b];
        }
    P.bed_c = ldc<CHAIN>(bed, i, j, ny, nx); P.bed_l = ldc<CHAIN>(bed, i, j - 1, ny, nx); P.bed_r = ldc<CHAIN>(bed, i, j + 1, ny, nx);
    P.bed_t = ldc<CHAIN>(bed, i - 1, j, ny, nx); P.bed_b = ldc<CHAIN>(bed, i + 1, j, ny, nx);
    P.beta_c = ldc<CHAIN>(beta, i, j, ny, nx); P.beta_l = ldc<CHAIN>(beta, i, j - 1, ny, nx); P.beta_r = ldc<CHAIN>(beta, i, j + 1, ny, nx);
    P.beta_t = ldc<CHAIN>(beta, i - 1, j, ny, nx); P.beta_b = ldc<CHAIN>(beta, i + 1, j, ny, nx);
    P.g_l = sigmoid(P.bed_l + rho_ratio<T>() * P.Hn[1][0], p.sig_c);
    P.g_r = sigmoid(P.bed_r + rho_ratio<T>() * P.Hn[1][2], p.sig_c);
    P.g_t = sigmoid(P.bed_t + rho_ratio<T>() * P.Hn[0][1], p.sig_c);
    P.g_b = sigmoid(P.bed_b + rho_ratio<T>() * P.Hn[2][1], p.sig_c);
    P.u_ll = W.u[r + 2][c];      P.u_rr = W.u[r + 2][c + 3];
    P.u_tl = W.u[r + 1][c + 1];  P.u_tr = W.u[r + 1][c + 2];
    P.u_bl = W.u[r + 3][c + 1];  P.u_br = W.u[r + 3][c + 2];
    P.v_lt = W.v[r + 1][c + 1];  P.v_lb = W.v[r + 2][c + 1];
    P.v_rt = W.v[r + 1][c + 3];  P.v_rb = W.v[r + 2][c + 3];
    P.v_tt = W.v[r][c + 2];      P.v_bb = W.v[r + 3][c + 2];
}

// Frozen per-cell coefficients of the forward local Newton loop: every term
// that depends only on neighbour values (fixed during a cell's iterations) is
// evaluated once here, so the loop only evaluates what depends on the cell's
// own 5 unknowns; the neighbour normal
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
// (terms of glide/cuda/vanka.cu:56-404; rows and columns u_l, u_r, v_t, v_b, H_c).
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

// State of a sweep, and where its kernel puts it: (u, v, H) plus the update of
// the sweep before from d (null: none), written to (ou, ov, oH) (null: not).
template <typename T> struct SweepState {
    const T *u, *v, *H, *d;
    T *ou, *ov, *oH;
    T omega;
};

// Per-cell Newton deltas.  scratch holds 5 cell arrays: 0.5*du_l, 0.5*du_r,
// 0.5*dv_t, 0.5*dv_b, dH.  FP64 has an instance for either local solve (PLAIN: not
// pivoted, gated sweeps only; a branch between them costs 3 %: 512^2, 10 pivoted
// steps 180 / 185 us), FP32 one for both.
template <typename T, bool LOCAL, bool PLAIN, typename P>
__global__ void __launch_bounds__(VX * VY, 4) vanka_cells_kernel(
    T* __restrict__ scratch, SweepState<T> q, const T* __restrict__ f_u, const T* __restrict__ f_v,
    const T* __restrict__ f_H, const T* __restrict__ bed, const T* __restrict__ B, const T* __restrict__ beta,
    const T* __restrict__ gamma, const int* __restrict__ flags, const int* __restrict__ any_active, int n_newton,
    T shift, T step, int pivot, int y0, Geo g, P p) {
    __shared__ Window<T> W;
    const int zero = chain_enter<true>();
    const int ny = g.ny, nx = g.nx;
    const int bz = blockIdx.z + zero;
    if (LOCAL && ld<true>(any_active + bz) == 0) return;
    f_u += bz * g.nu(); f_v += bz * g.nv();
    f_H += bz * g.nc(); bed += bz * g.nc(); B += bz * g.nc(); beta += bz * g.nc(); gamma += bz * g.nc();
    const int64_t nc = g.nc();
    scratch += bz * 5 * nc;
    if (LOCAL) flags += bz * int64_t(ny / REF_STRIDE + 1) * (nx / REF_STRIDE + 1);
    const int i0 = (blockIdx.y + y0) * VY + zero, j0 = blockIdx.x * VX;
    const int r = threadIdx.x / VX, c = threadIdx.x % VX;
    const int i = i0 + r, j = j0 + c;
    const bool has = q.d;
    const T* d = has ? q.d + bz * 5 * nc : q.H + bz * nc;
    const int64_t ds = has ? nc : 0;
    const State<T, LOCAL, true> st{q.u + bz * g.nu(), q.v + bz * g.nv(), q.H + bz * nc, d, d + ds, d + 2 * ds,
                                    d + 3 * ds, d + 4 * ds, flags, q.omega, ny, nx, has};
    T* ou = q.ou ? q.ou + bz * g.nu() : nullptr;
    T *ov = q.ov + bz * g.nv(), *oH = q.oH + bz * nc;
    const bool live = i < ny && j < nx && (!LOCAL || ref_tile_on<true>(flags, i, j, nx));
    if (LOCAL && !ou && !__syncthreads_or(live)) return;
    state_window(W, st, ou, ov, oH, i0, j0);
    if (LOCAL ? !__syncthreads_or(live) : (__syncthreads(), false)) return;   // nothing to solve
    eta_window<true>(W, B, i0, j0, ny, nx, p);
    __syncthreads();
    if (!live) return;

    Frozen<T> F;
    {
        Patch<T> pt;
        load_patch<true>(pt, W, r, c, bed, beta, i, j, ny, nx, p);
        make_frozen<T>(F, pt, ny, nx, p);
    }
    // 32-bit offsets within one field (the entry points bound a field below 2^31 elements)
    const int iu = i * (nx + 1) + j, ic32 = i * nx + j;
    const T ul0 = W.u[r + 2][c + 1], ur0 = W.u[r + 2][c + 2];
    const T vt0 = W.v[r + 1][c + 2], vb0 = W.v[r + 2][c + 2];
    const T H0 = W.H[r + 1][c + 1];
    const T fu_l = ld<true>(f_u + iu), fu_r = ld<true>(f_u + iu + 1);
    const T fv_t = ld<true>(f_v + ic32), fv_b = ld<true>(f_v + ic32 + nx);
    const T fH = ld<true>(f_H + ic32);
    const T thk = ld<true>(gamma + ic32);
    const T dti = T(1) / p.dt;
    T ul = ul0, ur = ur0, vt = vt0, vb = vb0, Hc = H0;
    for (int it = 0; it < n_newton; it++) {
        T J[25], rr[5], x[5];
        assemble_fast<T>(F, ul, ur, vt, vb, Hc, fu_l, fu_r, fv_t, fv_b, fH, thk, dti, p, J, rr);
        J[0] -= shift; J[6] -= shift; J[12] -= shift; J[18] -= shift; J[24] += shift;  // vanka.cu:406-410
        if (sizeof(T) == 8 ? !PLAIN : pivot != 0)
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

// (u, v, H) = (su, sv, sH) + omega * delta, face delta = sum of the two adjacent
// cells' halves; the source is the target itself or a copy of it.
template <typename T, bool LOCAL, bool CHAIN>
__global__ void vanka_apply_kernel(T* u, T* v, T* H, const T* su, const T* sv, const T* sH,
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
    su += bz * g.nu(); sv += bz * g.nv(); sH += bz * g.nc();
    scratch += bz * 5 * nc;
    if (LOCAL) flags += bz * int64_t(ny / REF_STRIDE + 1) * (nx / REF_STRIDE + 1);
    auto on = [&](int ii, int jj) { return !LOCAL || ref_tile_on<CHAIN>(flags, ii, jj, nx); };
    if (i < ny) {  // u-face (i,j), j in [0,nx]
        const int64_t k = int64_t(i) * (nx + 1) + j;
        T d = T(0);
        if (j < nx && on(i, j)) d += ld<CHAIN>(scratch + int64_t(i) * nx + j);                   // as u_l of cell (i,j)
        if (j > 0 && on(i, j - 1)) d += ld<CHAIN>(scratch + nc + int64_t(i) * nx + j - 1);        // as u_r of cell (i,j-1)
        u[k] = su[k] + omega * d;
    }
    if (j < nx) {  // v-face (i,j), i in [0,ny]
        const int64_t k = int64_t(i) * nx + j;
        T d = T(0);
        if (i < ny && on(i, j)) d += ld<CHAIN>(scratch + 2 * nc + k);
        if (i > 0 && on(i - 1, j)) d += ld<CHAIN>(scratch + 3 * nc + k - nx);
        v[k] = sv[k] + omega * d;
        if (i < ny) {
            T h = sH[k];
            if (on(i, j)) h += omega * ld<CHAIN>(scratch + 4 * nc + k);
            H[k] = h;
        }
    }
}

// --------------------------------------------------------------------------
// The cells' systems in arrow form, a thread per cell of a tile whose state and
// viscosities come from shared memory: stored for the linear sweeps (vanka_stored.cu
// has the march for large FP32 levels and the adjoint), or solved at once for one
// colour of the adjoint Vanka (glide/cuda/vanka.cu:441-840), for calls without
// room for stored systems.  Then lambda changes in place (within one colour every
// face has one writer) and half of the threads take a cell of the colour each:
// whole warps solve, the others are done.  One colour at 512^2, march / this: FP32
// 18.0 / 10.5 us, FP64 25.8 / 19.3; 256^2 9.8 / 5.0 and 13.7 / 6.2.
// --------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ Cell<T> patch_cell(const Patch<T>& P, T ul, T ur, T vt, T vb, int ny, int nx,
                                              const Phys<T>& p) {
    const T d2 = p.dxi * p.dxi, q = T(0.25) * d2, rr = rho_ratio<T>();
    const T wl = P.j > 0 ? T(1) : T(0), wr = P.j + 1 < nx ? T(1) : T(0);
    const T wt = P.i > 0 ? T(1) : T(0), wb = P.i + 1 < ny ? T(1) : T(0);
    T e[3][3];
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int b = 0; b < 3; b++) e[a][b] = P.eta[a][b] * P.Hn[a][b];
    auto surface = [&](T bed, T H) { return -(M<T>::max(bed, -rr * H) + H); };
    auto drag = [&](T g, T beta) { return T(0.5) * (g * beta + (T(1) - g) * p.water_drag); };
    Cell<T> C;
    C.H_1 = two(P.Hn[1][0], P.Hn[0][1]);
    C.H_2 = two(P.Hn[1][2], P.Hn[2][1]);
    C.Z_1 = two(surface(P.bed_l, C.H_1.x), surface(P.bed_t, C.H_1.y));
    C.Z_2 = two(surface(P.bed_r, C.H_2.x), surface(P.bed_b, C.H_2.y));
    C.B_1 = two(drag(P.g_l, P.beta_l), drag(P.g_t, P.beta_t));
    C.B_2 = two(drag(P.g_r, P.beta_r), drag(P.g_b, P.beta_b));
    C.bed = P.bed_c;
    C.beta = P.beta_c;
    C.n_1 = two(-ul, vt);
    C.n_2 = two(ur, -vb);
    C.D0 = two(ur - ul, vt - vb);
    C.E = T(2) * d2 * P.eta[1][1];
    const T e4 = q * P.eta[1][1];
    C.ew_p = two(e4 * wt * wl, e4 * wb * wr);
    C.ew_q = two(e4 * wb * wl, e4 * wt * wr);
    C.S_p = two(q * (e[0][0] + e[0][1] + e[1][0]) * wt * wl, q * (e[1][2] + e[2][1] + e[2][2]) * wb * wr);
    C.S_q = two(q * (e[1][0] + e[2][0] + e[2][1]) * wb * wl, q * (e[0][1] + e[0][2] + e[1][2]) * wt * wr);
    C.X_p = two((P.u_tl - ul) + (vt - P.v_lt), (ur - P.u_br) + (P.v_rb - vb));
    C.X_q = two((P.u_bl - ul) + (P.v_lb - vb), (ur - P.u_tr) + (vt - P.v_rt));
    C.K_1 = two(T(4) * d2 * e[1][0] * wl, T(4) * d2 * e[0][1] * wt);
    C.K_2 = two(T(4) * d2 * e[1][2] * wr, T(4) * d2 * e[2][1] * wb);
    C.W_1 = two(T(-0.5) * p.dxi * wl, T(-0.5) * p.dxi * wt);
    C.W_2 = two(T(-0.5) * p.dxi * wr, T(-0.5) * p.dxi * wb);
    C.f_H = C.thk = T(0);   // the active set is given
    return C;
}

template <typename T, int MODE, typename P>
__global__ void __launch_bounds__(VX * VY, 4) cell_systems_kernel(const StoredArgs<T> A, Geo g, P p) {
    __shared__ Window<T> W;
    const int zero = chain_enter<true>();
    const int ny = g.ny, nx = g.nx, bz = blockIdx.z + zero;
    const int64_t nc = g.nc();
    const T *u = A.u + bz * g.nu(), *v = A.v + bz * g.nv(), *H = A.H + bz * nc;
    const int i0 = (blockIdx.y + A.y0) * VY + zero, j0 = blockIdx.x * VX;
    const State<T, false, true> st{u, v, H, H, H, H, H, H, nullptr, T(0), ny, nx, false};
    state_window(W, st, (T*)nullptr, (T*)nullptr, (T*)nullptr, i0, j0);
    __syncthreads();
    eta_window<true>(W, A.B + bz * nc, i0, j0, ny, nx, p);
    __syncthreads();
    int r = threadIdx.x / VX, c = threadIdx.x % VX;
    if (MODE == SOLVE_ADJOINT) {
        r = threadIdx.x / (VX / 2);
        c = 2 * (threadIdx.x % (VX / 2)) + ((i0 + r + j0 + A.color) & 1);
    }
    const int i = i0 + r, j = j0 + c;
    if (r >= VY || i >= ny || j >= nx) return;
    const int64_t ic = i * nx + j;
    Patch<T> pt;
    load_patch<true>(pt, W, r, c, A.bed + bz * nc, A.beta + bz * nc, i, j, ny, nx, p);
    Cell<T> C = patch_cell<T>(pt, W.u[r + 2][c + 1], W.u[r + 2][c + 2], W.v[r + 1][c + 2], W.v[r + 2][c + 2], ny, nx, p);
    C.f_H = A.act ? T(0) : ld<true>(A.f_H + bz * nc + ic);
    C.thk = A.act ? T(0) : ld<true>(A.gamma + bz * nc + ic);
    Arrow<T> s;
    arrow_assemble<T>(C, W.H[r + 1][c + 1], A.shift, A.act ? (ld<true>(A.act + bz * nc + ic) > T(0.5) ? 1 : 0) : -1, p, s);
    if constexpr (MODE == STORE_LU) {
        store_matrix(A.out + bz * LU_ROOM * nc + ic, nc, s);
    } else {
        ArrowInv<T> q;
        arrow_factor<true>(transposed(s), q);
        adjoint_update<true>(q, A.ra_u + bz * g.nu(), A.ra_v + bz * g.nv(), A.ra_H + bz * nc, A.l_u + bz * g.nu(),
                             A.l_v + bz * g.nv(), A.l_H + bz * nc, i, j, nx, A.omega);
    }
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
static inline dim3 cell_grid(const Geo& g) { return dim3((g.nx + VX - 1) / VX, (g.ny + VY - 1) / VY, g.nb); }
static inline dim3 face_grid(const Geo& g) { return dim3((g.nx + 1 + 31) / 32, (g.ny + 1 + 7) / 8, g.nb); }

// Which form of the cell kernel: the tile, or the march (vanka_march.cu), whose
// cells cost less and whose warps need more of them: it pays from a size on that
// falls with the number of Newton steps and rises when only some rows are
// active.  The problem's own size decides, whatever its batch, because the two
// round differently.  So the FP32 FAS cycle keeps the tile at every size: a few
// FP32 cycles amplify a rounding 1e3 to 1e4 times, and a step's answer would move
// by up to 3e-4 between the forms.  Pivoted local solves exist in the tile only.
//
// Microseconds per sweep at both sides of the lines, tile / march; FP32 tile sweeps
// are one kernel each, FP64 ones two (room for one would be 34 MB more per level).
// FP32, 10 steps: 181^2 13.9 / 13.1, 256^2 14.6 / 15.0, 300^2 21.3 / 20.1, 512^2
// 45.4 / 43.3, 1024^2 172 / 142; 7 steps: 420^2 26.2 / 27.4, 600^2 48.9 / 47.1; 2 steps:
// 512^2 19.1 / 21.0, 600^2 25.7 / 27.3, 724^2 36.2 / 31.4, 1024^2 75.1 / 55.7.  FP64, the
// march: 10 steps: 32^2 17.4 / 14.9, 256^2 32.6 / 29.9, 1024^2 352 / 352; 2 steps: 32^2
// 9.7 / 9.7, 512^2 40.5 / 38.1, 1024^2 147 / 146.  Gated, a quarter (2 %) of the rows
// active, where the march's chunks of one or two rows repeat their preparatory rows or
// need a second wave: FP32, 2 steps: 512^2 13.6 / 20.1 (11.1 / 15.6), 724^2 24.0 / 27.9
// (18.6 / 20.2), 1024^2 44.8 / 36.3 (33.3 / 27.3); FP64, 2 steps: 256^2 15.0 / 14.4
// (13.9 / 13.5), 450^2 21.0 / 20.2 (17.5 / 19.7), 512^2 20.9 / 28.1 (16.2 / 20.1), 2048^2
// 235 / 281 (104 / 120); 10 steps: 450^2 38.1 / 34.2 (29.7 / 34.1), 512^2 38.3 / 52.5
// (26.3 / 34.1), 1024^2 116 / 118 (47.9 / 47.7), 2048^2 444 / 481 (125 / 141).
template <typename T>
static inline bool use_march(const Geo& g, int n_newton, bool gated, int pivot, bool cycle) {
    if (pivot) return false;
    const int64_t nc = g.nc(), k = int64_t(1) << 16;
    if constexpr (sizeof(T) == 8) return !gated || nc < 4 * k;
    if (cycle) return false;
    return nc >= (gated ? 8 * k : n_newton < 8 ? 6 * k : k);
}
// The update kernel of a sweep is chained while it fits the chip about once.
static inline bool apply_chained(const Geo& g) { return blocks_of(face_grid(g)) <= 592; }
template <typename T>
void run_march(const GlideLevelArgs*, const void*, const void*, const void*, int, double, double, const int*,
               const int*, void*, cudaStream_t);

template <typename T>
static SweepState<T> state_of(const GlideLevelArgs* a) {
    return {(const T*)a->u, (const T*)a->v, (const T*)a->H, nullptr, nullptr, nullptr, nullptr, T(0)};
}
template <typename T>
static void run_cells(const GlideLevelArgs* a, const void* f_u, const void* f_v, const void* f_H, int n_newton,
                      double shift, double step, int pivot, const int* flags, const int* any_active, void* scratch,
                      const Geo& g, bool cycle, const SweepState<T>& q, cudaStream_t s) {
    if (use_march<T>(g, n_newton, flags, pivot, cycle)) {
        run_march<T>(a, f_u, f_v, f_H, n_newton, shift, step, flags, any_active, scratch, s);
        return;
    }
    with_glen(a->params, make_phys<T>(a->params, a->dx, a->dt), [&](auto p) {
        using P = decltype(p);
        auto run = [&](auto kernel) {
            by_block_rows(cell_grid(g), [&](dim3 grid, int y0) {
                launch_chained<true>(kernel, grid, VX * VY, s, (T*)scratch, q, (const T*)f_u, (const T*)f_v,
                                     (const T*)f_H, (const T*)a->bed, (const T*)a->B, (const T*)a->beta,
                                     (const T*)a->gamma, flags, any_active, n_newton, T(shift), T(step), pivot, y0, g,
                                     p);
            });
        };
        if constexpr (sizeof(T) == 8) {
            if (!pivot) return run(vanka_cells_kernel<T, true, true, P>);   // gated: use_march
        }
        flags ? run(vanka_cells_kernel<T, true, false, P>) : run(vanka_cells_kernel<T, false, false, P>);
    });
}

// work (GLIDE_SWEEP_WORK elements, or null): a second state and a second set of
// cell arrays.  With them a sweep of the tile form is one kernel: it reads the
// state before and the update of the sweep before, and passes the sum on from
// one state to the other; one vanka_apply_kernel ends the call.  Microseconds per
// sweep of 10 Newton steps, two kernels / one: 32^2 8.1 / 6.7, 64^2 9.0 / 7.0,
// 256^2 16.1 / 14.1, 512^2 47.1 / 44.6, 1024^2 174 / 172; gated cycles gain most,
// a 512^2 step of three cycles 32.0 / 25.8 ms.
template <typename T>
int launch_vanka_sweeps(const GlideLevelArgs* a, const void* f_u, const void* f_v, const void* f_H, int n_iter,
                        int n_newton, double omega, double shift, const int* flags, const int* any_active,
                        void* scratch, cudaStream_t s, double newton_step, int pivot, bool cycle, void* work) {
    Geo g{a->ny, a->nx, a->nb};
    const bool chained = apply_chained(g), fused = work && !use_march<T>(g, n_newton, flags, pivot, cycle);
    SweepState<T> q = state_of<T>(a);
    q.omega = T(omega);
    T* const first[3] = {(T*)a->u, (T*)a->v, (T*)a->H};
    T *const wu = (T*)work, *const wv = wu + g.nu() * g.nb, *const wH = wv + g.nv() * g.nb;
    T* const second[3] = {wu, wv, wH};
    T *d = (T*)scratch, *d_next = fused ? wH + g.nc() * g.nb : d;
    auto apply = [&](auto chain) {
        constexpr bool CHAIN = decltype(chain)::value;
        auto run = [&](auto kernel) {
            launch_chained<CHAIN>(kernel, face_grid(g), dim3(32, 8), s, (T*)a->u, (T*)a->v, (T*)a->H, q.u, q.v, q.H,
                                  (const T*)d, flags, any_active, T(omega), g);
        };
        flags ? run(vanka_apply_kernel<T, true, CHAIN>) : run(vanka_apply_kernel<T, false, CHAIN>);
    };
    for (int k = 0; k < n_iter; k++) {
        run_cells<T>(a, f_u, f_v, f_H, n_newton, shift, newton_step, pivot, flags, any_active, d, g, cycle, q, s);
        if (!fused || k == n_iter - 1) {
            if (fused && q.ou) q.u = q.ou, q.v = q.ov, q.H = q.oH;
            chained ? apply(std::true_type{}) : apply(std::false_type{});
            continue;
        }
        if (q.ou) q.u = q.ou, q.v = q.ov, q.H = q.oH;   // this sweep's state; its update comes next
        T* const* to = q.u == first[0] ? second : first;
        q.ou = to[0], q.ov = to[1], q.oH = to[2];
        q.d = d;
        T* t = d; d = d_next; d_next = t;
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
        run_cells<T>(a, f_u, f_v, f_H, n_newton, shift, newton_step, 0, flags, any_active, scratch, g, false, state_of<T>(a), s);
    return (int)cudaGetLastError();
}

template <typename T, int MODE> int run_tile(const GlideLevelArgs* a, StoredArgs<T> A, cudaStream_t s) {
    Geo g{a->ny, a->nx, a->nb};
    A.u = (const T*)a->u; A.v = (const T*)a->v; A.H = (const T*)a->H;
    A.bed = (const T*)a->bed; A.B = (const T*)a->B; A.beta = (const T*)a->beta; A.gamma = (const T*)a->gamma;
    with_glen(a->params, make_phys<T>(a->params, a->dx, a->dt), [&](auto p) {
        by_block_rows(cell_grid(g), [&](dim3 grid, int y0) {
            A.y0 = y0;
            launch_chained<true>(cell_systems_kernel<T, MODE, decltype(p)>, grid, VX * VY, s, A, g, p);
        });
    });
    return (int)cudaGetLastError();
}

template <typename T>
int launch_vanka_adjoint(const GlideLevelArgs* a, void* l_u, void* l_v, void* l_H, const void* ra_u, const void* ra_v,
                         const void* ra_H, int color, double omega, cudaStream_t s) {
    StoredArgs<T> A{};
    A.act = (const T*)a->mask;
    A.l_u = (T*)l_u; A.l_v = (T*)l_v; A.l_H = (T*)l_H;
    A.ra_u = (const T*)ra_u; A.ra_v = (const T*)ra_v; A.ra_H = (const T*)ra_H;
    A.omega = T(omega);
    A.color = color;
    return run_tile<T, SOLVE_ADJOINT>(a, A, s);
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
                                        double, double, const int*, const int*, void*, cudaStream_t, double, int, bool, void*);\
    template int launch_vanka_cells<T>(const GlideLevelArgs*, const void*, const void*, const void*, int, int,     \
                                       double, const int*, const int*, void*, cudaStream_t, double);              \
    template int run_tile<T, STORE_LU>(const GlideLevelArgs*, StoredArgs<T>, cudaStream_t);                       \
    template int launch_vanka_adjoint<T>(const GlideLevelArgs*, void*, void*, void*, const void*, const void*,   \
                                         const void*, int, double, cudaStream_t);                                \
    template int launch_error_mask<T>(const GlideLevelArgs*, const void*, const void*, const void*, double,       \
                                      void*, int*, int*, cudaStream_t);                                           \
    template int launch_tile_flags<T>(const GlideLevelArgs*, const void*, int*, int*, cudaStream_t);
INST(float)
INST(double)
#undef INST

}  // namespace glide
