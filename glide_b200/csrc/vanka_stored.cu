// Vanka smoothers that form each cell's local matrix once: the linear sweeps of
// the defect correction and the adjoint smoother.
//
// Neither the state nor the active set changes while such a smoother runs, so
// the cells' 5x5 systems are formed once per call, in the arrow form of
// cell_system.cuh, and every sweep only solves them: 14 arrays for the linear
// sweep (bound by reading them: the factors of an unstructured elimination are
// 25), 18 for the adjoint (the solved form, without a reciprocal per sweep: its
// levels are small and wait on latency).
#include <type_traits>

#include "cell_system.cuh"

namespace glide {

constexpr int SW = 30;          // cell columns per warp of the march
constexpr int FC_NT = 128;
// --------------------------------------------------------------------------
// The march: a warp owns SW cell columns (lane l holds column j0 - 1 + l) and
// marches down a chunk of rows with the rows in reach in registers and the
// neighbouring columns in its lanes, as the residual does (ssa_stencil.cu).
// --------------------------------------------------------------------------
template <typename T, int MODE, typename P>
__global__ void __launch_bounds__(FC_NT, sizeof(T) == 4 ? 4 : 2)
    stored_cells_kernel(const StoredArgs<T> A, Geo g, P p) {
    const int ny = g.ny, nx = g.nx, b = blockIdx.y;
    const int wid = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
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

    const int strip = wid % A.n_strips, chunk = wid / A.n_strips;
    const int i0 = chunk * A.rows, i1 = min(i0 + A.rows, ny);
    const int jc = strip * SW - 1 + lane;
    const int jcc = clampi(jc, 0, nx - 1), juL = clampi(jc, 0, nx), juR = clampi(jc + 1, 0, nx);
    const int jvL = clampi(jc - 1, 0, nx - 1), jvR = clampi(jc + 1, 0, nx - 1);
    const bool first = lane == 0, last = lane == 31;
    const bool own = lane >= 1 && lane <= SW && jc < nx;
    const T dxi = p.dxi, d2 = p.dxi * p.dxi, rr = rho_ratio<T>();
    auto U = [&](int r, int col) -> T { return __ldg(u + (clampi(r, 0, ny - 1) * (nx + 1) + col)); };
    auto V = [&](int r, int col) -> T { return __ldg(v + (clampi(r, 0, ny) * nx + col)); };
    auto row = [&](const T* a, int r) -> T { return __ldg(a + (clampi(r, 0, ny - 1) * nx + jcc)); };

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

        if (i >= i0) {  // warp-uniform
            Cell<T> C;
            const T wl = jc > 0 ? T(1) : T(0), wr = jc + 1 < nx ? T(1) : T(0);
            const T wt = i > 0 ? T(1) : T(0), wb = i + 1 < ny ? T(1) : T(0);
            T umr = __shfl_down_sync(FULL, um, 1);
            if (last) umr = uRm;
            const T v0l = __shfl_up_sync(FULL, v0, 1), v0r = __shfl_down_sync(FULL, v0, 1);
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
            if (own) {
                const int ic = i * nx + jc;
                const T* act = A.act ? A.act + b * nc : nullptr;
                C.f_H = act ? T(0) : __ldg(A.f_H + b * nc + ic);
                C.thk = __ldg(A.gamma + b * nc + ic);
                Arrow<T> s;
                arrow_assemble<T>(C, Hc, A.shift, act ? (__ldg(act + ic) > T(0.5) ? 1 : 0) : -1, p, s);
                if constexpr (MODE == STORE_LU) {
                    store_matrix(A.out + b * LU_ROOM * nc + ic, nc, s);
                } else {
                    ArrowInv<T> q;
                    arrow_factor<true>(transposed(s), q);
                    store_solved(A.out + b * ADJ_N * nc + ic, nc, q);
                }
            }
        }
        // roll the window one row down
        um = u0; u0 = u1; u1 = u2; uRm = uR0; uR0 = uR1; uR1 = uR2;
        vm = v0; v0 = v1; v1 = v2; vL1 = vL2; vR1 = vR2;
        Hm = Hc; Zm = Zc; bm = bc; em = ec;
        Hc = Hp; Zc = Zp; bc = bp; ec = ep; etac = etap; bedc = bedp; betac = betap;
    }
}

// One colour of the adjoint sweep from stored factors: a thread per cell of the colour.
template <typename T, bool CHAIN>
__global__ void adjoint_color_kernel(const T* __restrict__ f, T* __restrict__ l_u, T* __restrict__ l_v,
                                     T* __restrict__ l_H, const T* __restrict__ ra_u, const T* __restrict__ ra_v,
                                     const T* __restrict__ ra_H, int color, T omega, int y0, Geo g) {
    const int ny = g.ny, nx = g.nx, b = blockIdx.z;
    const int i = (blockIdx.y + y0) * blockDim.y + threadIdx.y + chain_enter<CHAIN>();
    const int j = 2 * (blockIdx.x * blockDim.x + threadIdx.x) + ((i + color) & 1);
    if (i >= ny || j >= nx) return;
    const int64_t nc = g.nc();
    f += b * ADJ_N * nc + int64_t(i) * nx + j;
    T o[ADJ_N];
#pragma unroll
    for (int k = 0; k < ADJ_N; k++) o[k] = ld<CHAIN>(f + k * nc);
    ArrowInv<T> q;
    q.i = two(o[0], o[1]); q.w1 = two(o[2], o[3]); q.w2 = two(o[4], o[5]); q.Cd = two(o[6], o[7]);
    q.k = two(o[8], o[9]); q.e = two(o[10], o[11]);
    q.b11 = o[12]; q.b12 = o[13]; q.b22 = o[14]; q.ag = o[15]; q.bg = o[16]; q.ih = o[17];
    adjoint_update<CHAIN>(q, ra_u + b * g.nu(), ra_v + b * g.nv(), ra_H + b * nc, l_u + b * g.nu(), l_v + b * g.nv(),
                   l_H + b * nc, i, j, nx, omega);
}

// --------------------------------------------------------------------------
// One additive linear sweep, d += omega * sum of the cells' updates, in one
// pass.  A CTA owns 31 x 8 faces and solves 32 x 9 cells, the column to the
// left and the row above included: a face's two cells are this thread and its
// left neighbour (a shuffle) or the thread above (shared memory), so no cell
// array passes between two kernels.  A cell's solution needs nothing that
// another thread writes (the bound H + d_H >= gamma only enters its own d_H).
// Bound by reading the stored arrays; a thread per cell keeps all its loads in
// flight at once.  1021 x 1403, FP32, with its JVP: 115 us per sweep with 25
// factor arrays and two kernels, 105 as a march down the rows (3.5 TB/s), 94
// here.
// --------------------------------------------------------------------------
constexpr int LX = 31, LY = 8;

template <typename T>
__global__ void __launch_bounds__(32 * (LY + 1))
    vanka_linear_kernel(T* __restrict__ d_u, T* __restrict__ d_v, T* __restrict__ d_H, const T* __restrict__ lu,
                        const T* __restrict__ rho_u, const T* __restrict__ rho_v, const T* __restrict__ rho_H,
                        const T* __restrict__ H, const T* __restrict__ gamma, T omega, Geo g) {
    __shared__ T s_down[LY + 1][32];   // a cell's change of its lower face
    const int ny = g.ny, nx = g.nx, b = blockIdx.z;
    const int64_t nc = g.nc();
    d_u += b * g.nu(); d_v += b * g.nv(); d_H += b * nc;
    rho_u += b * g.nu(); rho_v += b * g.nv(); rho_H += b * nc; H += b * nc; gamma += b * nc;
    lu += b * LU_ROOM * nc;
    const int i = blockIdx.y * LY - 1 + threadIdx.y, j = blockIdx.x * LX - 1 + threadIdx.x;
    const bool cell = i >= 0 && i < ny && j >= 0 && j < nx;
    const bool own = threadIdx.x > 0 && threadIdx.y > 0;
    const int ic = i * nx + j, iu = i * (nx + 1) + j;
    Two<T> x1 = both(T(0)), x2 = both(T(0));   // outward changes of (l, t) and (r, b)
    T dH = T(0);
    if (cell) {
        const T* f = lu + ic;
        T o[LU_N];
#pragma unroll
        for (int k = 0; k < LU_N; k++) o[k] = __ldg(f + k * nc);
        const T ru_l = __ldg(rho_u + iu), ru_r = __ldg(rho_u + iu + 1);
        const T rv_t = __ldg(rho_v + ic), rv_b = __ldg(rho_v + ic + nx), rH = __ldg(rho_H + ic);
        const T room = own ? __ldg(gamma + ic) - __ldg(H + ic) - d_H[ic] : T(0);
        Arrow<T> s;
        s.D1 = two(o[0], o[1]); s.D2 = two(o[2], o[3]); s.p2 = o[4];
        s.c1 = two(o[5], o[6]); s.c2 = two(o[7], o[8]); s.e1 = two(o[9], o[10]); s.e2 = two(o[11], o[12]);
        s.j4 = o[13];
        s.hxy = both(T(0));
        ArrowInv<T> q;
        arrow_factor(s, q);
        T xh;
        arrow_solve(q, two(ru_l, -rv_t), two(-ru_r, rv_b), both(T(0)), T(0.5) * rH, x1, x2, xh);
        dH = M<T>::max(-xh, room);
        if (!(isfinite(x1.x) && isfinite(x1.y) && isfinite(x2.x) && isfinite(x2.y) && isfinite(xh))) {
            x1 = x2 = both(T(0));   // a failed local solve leaves its faces and its cell unchanged
            dH = T(0);
        }
    }
    // changes: u_l += x1.x/2, u_r -= x2.x/2, v_t -= x1.y/2, v_b += x2.y/2
    s_down[threadIdx.y][threadIdx.x] = x2.y;
    const T left = __shfl_up_sync(0xffffffffu, x2.x, 1);
    __syncthreads();
    if (!own || i > ny || j > nx) return;
    if (i < ny) d_u[iu] += omega * (T(0.5) * x1.x - T(0.5) * left);
    if (j < nx) d_v[ic] += omega * (T(0.5) * s_down[threadIdx.y - 1][threadIdx.x] - T(0.5) * x1.y);
    if (cell) d_H[ic] += omega * dH;
}

// --------------------------------------------------------------------------
// launchers
// --------------------------------------------------------------------------
// rows per warp and CTA size of a march over `lines` rows of n_strips strips
struct MarchShape {
    int rows, n_warps, threads;
    unsigned blocks;
};
// As few rows as fill the resident warps once.
static inline MarchShape march_shape(int n_strips, int lines, int nb, int warps_per_sm, int max_threads) {
    const int64_t units = int64_t(n_strips) * lines * nb;
    const int64_t rows = (units + 148 * warps_per_sm - 1) / (148 * warps_per_sm);
    MarchShape sh;
    sh.rows = int(rows > 64 ? 64 : rows);
    sh.n_warps = n_strips * ((lines + sh.rows - 1) / sh.rows);
    const int64_t per_sm = (int64_t(sh.n_warps) * nb + 147) / 148;
    sh.threads = 32 * int(per_sm < max_threads / 32 ? per_sm : max_threads / 32);
    sh.blocks = unsigned((sh.n_warps + sh.threads / 32 - 1) / (sh.threads / 32));
    return sh;
}

template <typename T, int MODE> int run_tile(const GlideLevelArgs*, StoredArgs<T>, cudaStream_t);   // vanka.cu

// Linear factors by the tile (vanka.cu), in FP32 from 2^18 cells of a problem on by
// the march; tile / march: FP32 256^2 3.9 / 4.8 us, 512^2 9.3 / 8.9, 1024^2 33.0 / 27.5;
// FP64 181^2 4.4 / 7.1, 256^2 5.8 / 7.4, 512^2 16.1 / 18.1, 1024^2 76 / 88.  The adjoint's by
// the march, which takes no shared memory: behind a kernel that does, its chained VJPs
// and colours run slower than the tile saves (40 sweeps at 256^2 FP64 1.39 / 1.20 ms,
// one by one; 1.15 / 1.16 ms from a graph).
template <typename T, int MODE>
static int run_stored(const GlideLevelArgs* a, StoredArgs<T> A, cudaStream_t s) {
    Geo g{a->ny, a->nx, a->nb};
    if constexpr (MODE == STORE_LU) {
        if (sizeof(T) == 8 || g.nc() < (int64_t(1) << 18)) return run_tile<T, MODE>(a, A, s);
    }
    A.u = (const T*)a->u; A.v = (const T*)a->v; A.H = (const T*)a->H;
    A.bed = (const T*)a->bed; A.B = (const T*)a->B; A.beta = (const T*)a->beta; A.gamma = (const T*)a->gamma;
    A.n_strips = (g.nx + SW - 1) / SW;
    const MarchShape sh = march_shape(A.n_strips, g.ny, g.nb, sizeof(T) == 4 ? 16 : 8, FC_NT);
    A.rows = sh.rows;
    A.n_warps = sh.n_warps;
    if constexpr (MODE != STORE_LU || sizeof(T) == 4)
        with_glen(a->params, make_phys<T>(a->params, a->dx, a->dt), [&](auto q) {
            launch_chained<false>(stored_cells_kernel<T, MODE, decltype(q)>, dim3(sh.blocks, g.nb), sh.threads, s, A, g,
                                  q);
        });
    return (int)cudaGetLastError();
}

// f_H null: the active set is the level's mask (glide_vanka_lu_masked)
template <typename T>
int launch_vanka_lu(const GlideLevelArgs* a, const void* f_H, void* lu, double shift, cudaStream_t s) {
    StoredArgs<T> A{};
    A.f_H = (const T*)f_H;
    A.act = f_H ? nullptr : (const T*)a->mask;
    A.out = (T*)lu;
    A.shift = T(shift);
    return run_stored<T, STORE_LU>(a, A, s);
}

// one sweep with a given rho = r + J d (recomputed by the caller in between)
template <typename T>
int launch_vanka_linear(const GlideLevelArgs* a, const void* rho_u, const void* rho_v, const void* rho_H,
                        const void* lu, void* d_u, void* d_v, void* d_H, double omega, cudaStream_t s) {
    Geo g{a->ny, a->nx, a->nb};
    const dim3 grid((g.nx + 1 + LX - 1) / LX, (g.ny + 1 + LY - 1) / LY, g.nb);
    launch_chained<false>(
        vanka_linear_kernel<T>, grid, dim3(32, LY + 1), s, (T*)d_u, (T*)d_v, (T*)d_H, (const T*)lu, (const T*)rho_u, (const T*)rho_v, (const T*)rho_H, (const T*)a->H,
        (const T*)a->gamma, T(omega), g);
    return (int)cudaGetLastError();
}

template <typename T> int launch_adjoint_factors(const GlideLevelArgs* a, void* factors, cudaStream_t s) {
    StoredArgs<T> A{};
    A.act = (const T*)a->mask;
    A.out = (T*)factors;
    return run_stored<T, STORE_ADJOINT>(a, A, s);
}

template <typename T>
int launch_adjoint_color(const GlideLevelArgs* a, const void* factors, void* l_u, void* l_v, void* l_H,
                         const void* ra_u, const void* ra_v, const void* ra_H, int color, double omega,
                         cudaStream_t s) {
    Geo g{a->ny, a->nx, a->nb};
    const dim3 blk(32, 4), grd(((g.nx + 1) / 2 + 31) / 32, (g.ny + 3) / 4, g.nb);
    auto go = [&](auto chain) {
        constexpr bool CHAIN = decltype(chain)::value;
        by_block_rows(grd, [&](dim3 grid, int y0) {
            launch_chained<CHAIN>(adjoint_color_kernel<T, CHAIN>, grid, blk, s, (const T*)factors, (T*)l_u, (T*)l_v,
                                  (T*)l_H, (const T*)ra_u, (const T*)ra_v, (const T*)ra_H, color, T(omega), y0, g);
        });
    };
    blocks_of(grd) <= 592 ? go(std::true_type{}) : go(std::false_type{});
    return (int)cudaGetLastError();
}

#define INST(T)                                                                                                     \
    template int launch_vanka_lu<T>(const GlideLevelArgs*, const void*, void*, double, cudaStream_t);               \
    template int launch_vanka_linear<T>(const GlideLevelArgs*, const void*, const void*, const void*, const void*,  \
                                        void*, void*, void*, double, cudaStream_t);                                 \
    template int launch_adjoint_factors<T>(const GlideLevelArgs*, void*, cudaStream_t);                             \
    template int launch_adjoint_color<T>(const GlideLevelArgs*, const void*, void*, void*, void*, const void*,      \
                                         const void*, const void*, int, double, cudaStream_t);
INST(float)
INST(double)
#undef INST

}  // namespace glide
