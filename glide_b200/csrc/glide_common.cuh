// Shared device code for the SSA hot path on B200 (sm_100a).
//
// Physics follows the reference discretisation (glide/cuda/stress.cu,
// glide/cuda/flux.cu, glide/cuda/viscosity.cu); every term returns its value
// together with the partial derivatives the solvers need, written as plain
// value-plus-partials structs instead of the reference's dual numbers.
// Everything is templated on the working precision T (float or double).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "glide_b200.h"

namespace glide {

// host-side count of kernel launches issued by this library (also counts
// launches recorded during stream capture); see glide_launch_count
void count_launch();
long long launch_total();

// --------------------------------------------------------------------------
// Chained launches.  A smoother is a chain of short kernels, each reading what
// the one before wrote; between two of them the chip idles for the launch.  A
// kernel launched with launch_chained() may start while its predecessor still
// runs (programmatic stream serialization); chain_enter<true>(), its first
// statement, lets its own successor do the same and then waits until the
// predecessor has completed and its writes are visible.  Every thread of such
// a kernel calls it before its first access, so completion is transitive along
// the chain.  The predecessor's writes fall into the kernel's lifetime, so it
// must not read them through the read-only path: ld<true>() loads without it,
// and indices take chain_enter()'s zero, which keeps the compiler from moving
// a load above the wait.  200 sweeps of a 32^2 level, launched one by one: 2.87 ms
// plain, 2.17 ms chained.  The marches and the updates that fill the chip gain
// nothing and run with CHAIN = false and read-only loads (2-3 % faster there); the
// tiles, which load a window at once, are chained at every size (FP32 sweeps of
// 1024^2 with 2 / 10 Newton steps 76.6 / 174.6 us, 82.6 / 177.4 unchained).
// --------------------------------------------------------------------------
template <bool CHAIN> __device__ __forceinline__ int chain_enter() {
    if constexpr (!CHAIN) return 0;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    int zero = 0;
    asm volatile("" : "+r"(zero)::"memory");
    return zero;
}
template <bool CHAIN, typename T> __device__ __forceinline__ T ld(const T* p) {
    if constexpr (CHAIN)
        return __ldca(p);
    else
        return __ldg(p);
}

template <bool CHAIN, typename... KA, typename... A>
inline void launch_chained(void (*kernel)(KA...), dim3 grid, dim3 block, cudaStream_t s, A&&... args) {
    count_launch();
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    if constexpr (CHAIN) {
        // a captured graph issues its kernels back to back by itself (32^2: 8.1 us per sweep either way)
        cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
        cudaStreamIsCapturing(s, &st);
        c.numAttrs = st == cudaStreamCaptureStatusNone ? 1 : 0;
    }
    cudaLaunchKernelEx(&c, kernel, KA(args)...);
}
// A launch has at most 65,535 rows of blocks: taller grids go in pieces, each
// told the block row it starts at.
template <typename F> inline void by_block_rows(dim3 grid, F&& launch) {
    for (unsigned y0 = 0; y0 < grid.y; y0 += 65535u)
        launch(dim3(grid.x, grid.y - y0 < 65535u ? grid.y - y0 : 65535u, grid.z), int(y0));
}
static inline int64_t blocks_of(dim3 g) { return int64_t(g.x) * g.y * g.z; }

// --------------------------------------------------------------------------
// precision helpers
// --------------------------------------------------------------------------
template <typename T> struct M;
// FP32 exp/pow: the hardware approximations by default, as the reference's
// --use_fast_math build of its ice kernels uses (glide/kernels.py:72);
// -DGLIDE_FP32_ACCURATE_MATH=1 selects expf/powf and IEEE division.
#ifndef GLIDE_FP32_ACCURATE_MATH
#define GLIDE_FP32_ACCURATE_MATH 0
#endif
template <> struct M<float> {
#if GLIDE_FP32_ACCURATE_MATH
    static __device__ __forceinline__ float exp(float x) { return expf(x); }
    static __device__ __forceinline__ float pow(float x, float y) { return powf(x, y); }
    static __device__ __forceinline__ float rcp(float x) { return 1.0f / x; }
#else
    static __device__ __forceinline__ float exp(float x) { return __expf(x); }
    static __device__ __forceinline__ float pow(float x, float y) { return __powf(x, y); }
    // reciprocal of the LU pivots and of the sigmoid denominator: the fast
    // approximate division, as the reference's fast-math build divides
    static __device__ __forceinline__ float rcp(float x) { return __fdividef(1.0f, x); }
#endif
    static __device__ __forceinline__ float sqrt(float x) { return sqrtf(x); }
    static __device__ __forceinline__ float abs(float x) { return fabsf(x); }
    static __device__ __forceinline__ float copysign(float a, float b) { return copysignf(a, b); }
    static __device__ __forceinline__ float max(float a, float b) { return fmaxf(a, b); }
    static __device__ __forceinline__ float min(float a, float b) { return fminf(a, b); }
};
template <> struct M<double> {
    static __device__ __forceinline__ double exp(double x) { return ::exp(x); }
    static __device__ __forceinline__ double pow(double x, double y) { return ::pow(x, y); }
    static __device__ __forceinline__ double sqrt(double x) { return ::sqrt(x); }
    static __device__ __forceinline__ double rcp(double x) { return 1.0 / x; }
    static __device__ __forceinline__ double abs(double x) { return fabs(x); }
    static __device__ __forceinline__ double copysign(double a, double b) { return ::copysign(a, b); }
    static __device__ __forceinline__ double max(double a, double b) { return fmax(a, b); }
    static __device__ __forceinline__ double min(double a, double b) { return fmin(a, b); }
};

// rho_ice / rho_water, as in glide/cuda/stress.cu:250
template <typename T> __device__ __forceinline__ T rho_ratio() { return T(0.917); }

// Physical parameters converted to the working precision.
template <typename T> struct Phys {
    T glen_exp;      // (1-n)/(2n)
    T eps_reg, water_drag, calving_rate, sig_c;
    int gl_deriv;
    T dx, dxi, dt;
};

// Glen's exponent n = 3 in FP64: the viscosity's power is a reciprocal cube
// root, several times cheaper than the general pow (which is most of an FP64
// stencil's instructions) and as accurate.  The kernels are instantiated for
// both; FP32's pow is two hardware approximations either way.  FP64 VJP at
// 1024^2 with the gradient of beta: 159 us with pow, 129 with the cube root.
template <typename T> struct PhysCube : Phys<T> {
    explicit PhysCube(const Phys<T>& p) : Phys<T>(p) {}
};
template <typename T> __device__ __forceinline__ T glen_pow(T x, const Phys<T>& p) {
    return M<T>::pow(x, p.glen_exp);
}
__device__ __forceinline__ double glen_pow(double x, const PhysCube<double>&) { return ::rcbrt(x); }
// go(p) with the parameters in the type the kernels should be instantiated for
template <typename T, typename F> inline void with_glen(const GlidePhysicsParams& gp, const Phys<T>& p, F&& go) {
    if constexpr (sizeof(T) == 8) {
        if (gp.n == 3.0) {
            go(PhysCube<T>(p));
            return;
        }
    }
    go(p);
}

template <typename T>
inline Phys<T> make_phys(const GlidePhysicsParams& p, double dx, double dt) {
    Phys<T> q;
    T n = T(p.n);
    q.glen_exp = (T(1) - n) / (T(2) * n);
    q.eps_reg = T(p.eps_reg);
    q.water_drag = T(p.water_drag);
    q.calving_rate = T(p.calving_rate);
    q.sig_c = T(p.gl_sigmoid_c);
    q.gl_deriv = p.gl_derivatives;
    q.dx = T(dx);
    q.dxi = T(1) / T(dx);
    q.dt = T(dt);
    return q;
}

// Geometry of one level (batch of nb independent problems).
struct Geo {
    int ny, nx, nb;
    __host__ __device__ int64_t nu() const { return int64_t(ny) * (nx + 1); }
    __host__ __device__ int64_t nv() const { return int64_t(ny + 1) * nx; }
    __host__ __device__ int64_t nc() const { return int64_t(ny) * nx; }
};

__device__ __forceinline__ int clampi(int x, int lo, int hi) { return x < lo ? lo : (x > hi ? hi : x); }

// --------------------------------------------------------------------------
// clamped access to a cell field (same semantics as glide/cuda/common.cu:78-125:
// every index is clamped to the field's own extent).  Offsets are 32-bit
// element counts: the entry points reject problems whose fields reach 2^31
// elements (GLIDE_E_TOO_LARGE).
// --------------------------------------------------------------------------
template <bool CHAIN = false, typename T>
__device__ __forceinline__ T ldc(const T* __restrict__ a, int i, int j, int ny, int nx) {
    return ld<CHAIN>(a + (clampi(i, 0, ny - 1) * nx + clampi(j, 0, nx - 1)));
}

// --------------------------------------------------------------------------
// local terms (value + partials)
// --------------------------------------------------------------------------
template <typename T> __device__ __forceinline__ T sigmoid(T z, T c) {
    T s = M<T>::min(M<T>::max(c * z, T(-20)), T(20));   // common.cu:67-70
    return M<T>::rcp(T(1) + M<T>::exp(-s));
}

// Normal stress on a cell (stress.cu:43-102).  XX: 2 etaH (2 ux + vy);
// YY: 2 etaH (ux + 2 vy).  Zero when the cell is outside the domain.
template <typename T> struct NormalStress {
    T res, d_ul, d_ur, d_vt, d_vb, d_etaH;
};
template <typename T, bool XX>
__device__ __forceinline__ NormalStress<T> normal_stress(T ul, T ur, T vt, T vb, T etaH, T dxi, bool valid) {
    NormalStress<T> o;
    T pre = T(2) * etaH * dxi;
    T e = XX ? (T(2) * (ur - ul) * dxi + (vt - vb) * dxi) : ((ur - ul) * dxi + T(2) * (vt - vb) * dxi);
    T w = valid ? T(1) : T(0);
    o.res = T(2) * etaH * e * w;
    o.d_ul = (XX ? T(-2) : T(-1)) * pre * w;
    o.d_ur = (XX ? T(2) : T(1)) * pre * w;
    o.d_vt = (XX ? T(1) : T(2)) * pre * w;
    o.d_vb = (XX ? T(-1) : T(-2)) * pre * w;
    o.d_etaH = T(2) * e * w;
    return o;
}

// Shear stress on a vertex (stress.cu:159-183): 2 etaH eps_xy, zero on boundary vertices.
template <typename T> struct ShearStress {
    T res, d_ut, d_ub, d_vl, d_vr, d_etaH;
};
template <typename T>
__device__ __forceinline__ ShearStress<T> shear_stress(T ut, T ub, T vl, T vr, T etaH, T dxi, bool valid) {
    ShearStress<T> o;
    T w = valid ? T(1) : T(0);
    T exy = T(0.5) * ((ut - ub) * dxi + (vr - vl) * dxi);
    T pre = etaH * dxi * w;
    o.res = T(2) * etaH * exy * w;
    o.d_ut = pre;
    o.d_ub = -pre;
    o.d_vl = -pre;
    o.d_vr = pre;
    o.d_etaH = T(2) * exy * w;
    return o;
}

// Basal drag between cells 1 and 2 of a face (stress.cu:244-276, :330-361).
template <typename T> struct BasalDrag {
    T res, d_vel, d_H1, d_H2, d_beta1, d_beta2;
};
// The drag of a face from the grounded fractions of its two cells (the Vanka
// loop hoists the neighbour's sigmoid out of its Newton iterations).
template <typename T>
__device__ __forceinline__ BasalDrag<T> basal_drag_g(T vel, T g1, T g2, T beta1, T beta2, const Phys<T>& p) {
    BasalDrag<T> o;
    T be = T(0.5) * ((g1 * beta1 + (T(1) - g1) * p.water_drag) + (g2 * beta2 + (T(1) - g2) * p.water_drag));
    o.res = -be * vel;
    o.d_vel = -be;
    o.d_beta1 = T(-0.5) * g1 * vel;
    o.d_beta2 = T(-0.5) * g2 * vel;
    o.d_H1 = T(0);
    o.d_H2 = T(0);
    if (p.gl_deriv) {
        T s1 = p.sig_c * g1 * (T(1) - g1), s2 = p.sig_c * g2 * (T(1) - g2);
        o.d_H1 = T(-0.5) * (rho_ratio<T>() * s1) * (beta1 - p.water_drag) * vel;
        o.d_H2 = T(-0.5) * (rho_ratio<T>() * s2) * (beta2 - p.water_drag) * vel;
    }
    return o;
}

// Upwind face flux (flux.cu:39-64, :110-135).  For x-faces a = left cell,
// b = right cell, q = H_avg u - 0.5|u|(H_b - H_a).  For y-faces a = bottom
// (row i), b = top (row i-1), q = H_avg v - 0.5|v|(H_top - H_bottom).
template <typename T> struct Flux {
    T res, d_vel, d_Ha, d_Hb;
};
template <typename T> __device__ __forceinline__ Flux<T> upwind_flux(T vel, T Ha, T Hb, bool valid) {
    Flux<T> o;
    T w = valid ? T(1) : T(0);
    T Havg = T(0.5) * (Ha + Hb);
    T m = M<T>::abs(vel);
    T s = M<T>::copysign(T(1), vel);
    o.res = (Havg * vel - T(0.5) * m * (Hb - Ha)) * w;
    o.d_vel = (Havg - T(0.5) * s * (Hb - Ha)) * w;
    o.d_Ha = T(0.5) * (vel + m) * w;
    o.d_Hb = T(0.5) * (vel - m) * w;
    return o;
}

// Calving sink -c (1-g) H (flux.cu:187-211).
template <typename T> struct Calving {
    T res, d_H;
};
template <typename T> __device__ __forceinline__ Calving<T> calving_g(T H, T g, const Phys<T>& p) {
    Calving<T> o;
    o.res = -p.calving_rate * (T(1) - g) * H;
    o.d_H = -p.calving_rate * (T(1) - g);
    if (p.gl_deriv) o.d_H += p.calving_rate * H * (rho_ratio<T>() * (p.sig_c * g * (T(1) - g)));
    return o;
}

// Cell viscosity from its 4 faces and the 8 neighbouring faces of the 4
// corner shear rates (viscosity.cu:61-112); optional tangent (viscosity.cu:4-59).
template <typename T> struct EtaIn {
    T ul, ur, vt, vb;             // own faces
    T u_tl, u_tr, u_bl, u_br;     // u at (i-1,j), (i-1,j+1), (i+1,j), (i+1,j+1)
    T v_lt, v_rt, v_lb, v_rb;     // v at (i,j-1), (i,j+1), (i+1,j-1), (i+1,j+1)
};
template <typename T> struct EtaOut {
    T eta, eII, exy[4], ux, vy;
};
template <typename T, typename P>
__device__ __forceinline__ EtaOut<T> cell_eta(const EtaIn<T>& a, T Bc, int i, int j, int ny, int nx, const P& p) {
    EtaOut<T> o;
    T dxi = p.dxi;
    o.ux = (a.ur - a.ul) * dxi;
    o.vy = (a.vt - a.vb) * dxi;
    T mtl = (i > 0 && j > 0) ? T(1) : T(0);
    T mtr = (i > 0 && j < nx - 1) ? T(1) : T(0);
    T mbl = (i < ny - 1 && j > 0) ? T(1) : T(0);
    T mbr = (i < ny - 1 && j < nx - 1) ? T(1) : T(0);
    o.exy[0] = T(0.5) * ((a.u_tl - a.ul) * dxi + (a.vt - a.v_lt) * dxi) * mtl;
    o.exy[1] = T(0.5) * ((a.u_tr - a.ur) * dxi + (a.v_rt - a.vt) * dxi) * mtr;
    o.exy[2] = T(0.5) * ((a.ul - a.u_bl) * dxi + (a.vb - a.v_lb) * dxi) * mbl;
    o.exy[3] = T(0.5) * ((a.ur - a.u_br) * dxi + (a.v_rb - a.vb) * dxi) * mbr;
    T e2 = T(0.25) * (o.exy[0] * o.exy[0] + o.exy[1] * o.exy[1] + o.exy[2] * o.exy[2] + o.exy[3] * o.exy[3]);
    o.eII = o.ux * o.ux + o.vy * o.vy + o.ux * o.vy + e2 + p.eps_reg;
    o.eta = T(0.5) * Bc * glen_pow(o.eII, p);
    return o;
}
// Tangent of eta for a tangent (du, dv) of the same 12 faces.  FP64 takes it from
// eta (a quarter of the error of a second power, which costs as much as the rest
// of the row); FP32's power is two hardware approximations, and one of its own
// keeps its error apart from eta's.
template <typename T>
__device__ __forceinline__ T cell_eta_tangent(const EtaOut<T>& e, const EtaIn<T>& d, T Bc, int i, int j, int ny, int nx,
                                              const Phys<T>& p) {
    T dxi = p.dxi;
    T dux = (d.ur - d.ul) * dxi;
    T dvy = (d.vt - d.vb) * dxi;
    T mtl = (i > 0 && j > 0) ? T(1) : T(0);
    T mtr = (i > 0 && j < nx - 1) ? T(1) : T(0);
    T mbl = (i < ny - 1 && j > 0) ? T(1) : T(0);
    T mbr = (i < ny - 1 && j < nx - 1) ? T(1) : T(0);
    T de0 = T(0.5) * ((d.u_tl - d.ul) * dxi + (d.vt - d.v_lt) * dxi) * mtl;
    T de1 = T(0.5) * ((d.u_tr - d.ur) * dxi + (d.v_rt - d.vt) * dxi) * mtr;
    T de2 = T(0.5) * ((d.ul - d.u_bl) * dxi + (d.vb - d.v_lb) * dxi) * mbl;
    T de3 = T(0.5) * ((d.ur - d.u_br) * dxi + (d.v_rb - d.vb) * dxi) * mbr;
    T de2sum = T(0.25) * (T(2) * e.exy[0] * de0 + T(2) * e.exy[1] * de1 + T(2) * e.exy[2] * de2 +
                          T(2) * e.exy[3] * de3);
    T deII = T(2) * e.ux * dux + T(2) * e.vy * dvy + (e.ux * dvy + e.vy * dux) + de2sum;
    if constexpr (sizeof(T) == 4) return T(0.5) * Bc * (p.glen_exp * M<T>::pow(e.eII, p.glen_exp - T(1)) * deII);
    return p.glen_exp * e.eta * (deII * M<T>::rcp(e.eII));   // eta ~ eII^glen_exp
}

}  // namespace glide
