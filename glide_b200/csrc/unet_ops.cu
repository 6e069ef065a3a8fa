// Data-movement kernels around the tensor-core GEMM for the learned guess:
// im2col of a 3x3 "same" convolution, its transpose (col2im, gather form so
// every output has one writer), BF16 transposes, and the pack/unpack between
// the solver's staggered fields and the network's NHWC tensors.
#include <cuda_bf16.h>
#include <stdint.h>

#include "glide_b200.h"

namespace glide {
void count_launch();
}

namespace glide {

// col[p, (ky*3+kx)*C + c] = x[b, y+ky-1, x+kx-1, c] (zero outside); p = (b*H + y)*W + x.
// Columns [9C, Kp) are zero.
__global__ void im2col3_k(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ col, int Bn, int H, int W,
                          int C, int Kp) {
    const int64_t total = int64_t(Bn) * H * W * Kp;
    for (int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; idx < total;
         idx += int64_t(gridDim.x) * blockDim.x) {
        const int k = int(idx % Kp);
        const int64_t p = idx / Kp;
        __nv_bfloat16 v = __float2bfloat16(0.0f);
        if (k < 9 * C) {
            const int tap = k / C, c = k % C;
            const int ky = tap / 3, kx = tap % 3;
            const int xx = int(p % W), yy = int((p / W) % H), b = int(p / (int64_t(W) * H));
            const int sy = yy + ky - 1, sx = xx + kx - 1;
            if (sy >= 0 && sy < H && sx >= 0 && sx < W) v = x[((int64_t(b) * H + sy) * W + sx) * C + c];
        }
        col[idx] = v;
    }
}

// dx[b,y,x,c] = sum_{ky,kx} dcol[p(b, y-ky+1, x-kx+1), (ky*3+kx)*C + c]
__global__ void col2im3_k(const float* __restrict__ dcol, float* __restrict__ dx, int Bn, int H, int W, int C, int Kp) {
    const int64_t total = int64_t(Bn) * H * W * C;
    for (int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; idx < total;
         idx += int64_t(gridDim.x) * blockDim.x) {
        const int c = int(idx % C);
        const int64_t pix = idx / C;
        const int xx = int(pix % W), yy = int((pix / W) % H), b = int(pix / (int64_t(W) * H));
        float acc = 0.0f;
#pragma unroll
        for (int ky = 0; ky < 3; ky++) {
#pragma unroll
            for (int kx = 0; kx < 3; kx++) {
                const int oy = yy - ky + 1, ox = xx - kx + 1;
                if (oy >= 0 && oy < H && ox >= 0 && ox < W) {
                    const int64_t p = (int64_t(b) * H + oy) * W + ox;
                    acc += dcol[p * Kp + (ky * 3 + kx) * C + c];
                }
            }
        }
        dx[idx] = acc;
    }
}

// dst[c, r] = src[r, c]  (R x Cc -> Cc x R), BF16, 32x32 smem tiles
__global__ void transpose_bf16_k(const __nv_bfloat16* __restrict__ src, __nv_bfloat16* __restrict__ dst, int R,
                                 int Cc) {
    __shared__ __nv_bfloat16 t[32][33];
    const int r0 = blockIdx.y * 32, c0 = blockIdx.x * 32;
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
        const int r = r0 + k, c = c0 + threadIdx.x;
        t[k][threadIdx.x] = (r < R && c < Cc) ? src[int64_t(r) * Cc + c] : __float2bfloat16(0.0f);
    }
    __syncthreads();
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
        const int c = c0 + k, r = r0 + threadIdx.x;
        if (c < Cc && r < R) dst[int64_t(c) * R + r] = t[threadIdx.x][k];
    }
}

// 2x2 average, 8 channels per thread (glide_b200.guess._pool in one pass)
__global__ void pool2_k(const uint4* __restrict__ x, uint4* __restrict__ y, int Ho, int Wo, int C8, int64_t total) {
    const int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const int c = int(idx % C8);
    const int64_t p = idx / C8;
    const int xo = int(p % Wo);
    const int64_t row = p / Wo;   // image and output row
    const uint4* s = x + ((2 * row) * (2 * Wo) + 2 * xo) * C8 + c;
    const int64_t down = int64_t(2 * Wo) * C8;
    const uint4 q[4] = {__ldg(s), __ldg(s + C8), __ldg(s + down), __ldg(s + down + C8)};
    __align__(16) __nv_bfloat16 h[8];
#pragma unroll
    for (int e = 0; e < 8; e++) {
        float v[4];
#pragma unroll
        for (int k = 0; k < 4; k++) v[k] = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(&q[k])[e]);
        h[e] = __float2bfloat16(((v[0] + v[1]) + (v[2] + v[3])) * 0.25f);
    }
    y[idx] = *reinterpret_cast<const uint4*>(h);
}

// Network input of one cell per thread: H/1000, bed/1000, (log beta + 2.2)/0.7,
// B/35 and four zeros, BF16.  Same roundings as glide_b200.guess.features in
// torch (FP32, division by a constant as the product with its reciprocal).
template <typename T>
__global__ void guess_features_k(const T* __restrict__ H, const T* __restrict__ bed, const T* __restrict__ beta,
                                 const T* __restrict__ B, uint4* __restrict__ x, int64_t n) {
    const int64_t k = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (k >= n) return;
    float b = float(beta[k]);
    b = b < 1e-8f ? 1e-8f : b;
    const float f[4] = {__fmul_rn(float(H[k]), 1.0f / 1000.0f), __fmul_rn(float(bed[k]), 1.0f / 1000.0f),
                        __fmul_rn(__fadd_rn(logf(b), 2.2f), 1.0f / 0.7f), __fmul_rn(float(B[k]), 1.0f / 35.0f)};
    __align__(16) __nv_bfloat16 h[8];
#pragma unroll
    for (int e = 0; e < 8; e++) h[e] = __float2bfloat16(e < 4 ? f[e & 3] : 0.0f);
    x[k] = *reinterpret_cast<const uint4*>(h);
}

// Cell velocities (ny, nx, 2) in units of scale -> staggered u (ny, nx+1) and v
// (ny+1, nx) in FP64: FP32 averages of the two cells of a face, the cell's own
// value on the boundary (glide_b200.guess.faces_from_cells in one pass).
__global__ void guess_faces_k(const float2* __restrict__ p, double* __restrict__ u, double* __restrict__ v, int ny,
                              int nx, float scale) {
    const int b = blockIdx.z, j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y * blockDim.y + threadIdx.y;
    if (i > ny || j > nx) return;
    p += int64_t(b) * ny * nx;
    u += int64_t(b) * ny * (nx + 1);
    v += int64_t(b) * (ny + 1) * nx;
    auto face = [&](float a, float c) {
        return double(__fmul_rn(0.5f, __fadd_rn(__fmul_rn(c, scale), __fmul_rn(a, scale))));
    };
    if (i < ny) {
        const float2* r = p + int64_t(i) * nx;
        u[int64_t(i) * (nx + 1) + j] = j == 0    ? double(__fmul_rn(r[0].x, scale))
                                       : j == nx ? double(__fmul_rn(r[nx - 1].x, scale))
                                                 : face(r[j - 1].x, r[j].x);
    }
    if (j < nx) {
        const float2* c = p + j;
        v[int64_t(i) * nx + j] = i == 0    ? double(__fmul_rn(c[0].y, scale))
                                 : i == ny ? double(__fmul_rn(c[int64_t(ny - 1) * nx].y, scale))
                                           : face(c[int64_t(i - 1) * nx].y, c[int64_t(i) * nx].y);
    }
}

static inline unsigned blocks_for(int64_t n) {
    int64_t b = (n + 255) / 256;
    return unsigned(b > 148 * 64 ? 148 * 64 : (b < 1 ? 1 : b));
}

}  // namespace glide

extern "C" int glide_im2col3_bf16(const void* x, void* col, int Bn, int H, int W, int C, int Kp, void* stream) {
    if (!x || !col) return GLIDE_E_NULL;
    if (Bn < 1 || H < 1 || W < 1 || C < 1 || Kp < 9 * C) return GLIDE_E_SHAPE;
    glide::count_launch(), glide::im2col3_k<<<glide::blocks_for(int64_t(Bn) * H * W * Kp), 256, 0, (cudaStream_t)stream>>>(
        (const __nv_bfloat16*)x, (__nv_bfloat16*)col, Bn, H, W, C, Kp);
    return (int)cudaGetLastError();
}

extern "C" int glide_col2im3_f32(const float* dcol, float* dx, int Bn, int H, int W, int C, int Kp, void* stream) {
    if (!dcol || !dx) return GLIDE_E_NULL;
    if (Bn < 1 || H < 1 || W < 1 || C < 1 || Kp < 9 * C) return GLIDE_E_SHAPE;
    glide::count_launch(), glide::col2im3_k<<<glide::blocks_for(int64_t(Bn) * H * W * C), 256, 0, (cudaStream_t)stream>>>(dcol, dx, Bn, H, W,
                                                                                                   C, Kp);
    return (int)cudaGetLastError();
}

extern "C" int glide_transpose_bf16(const void* src, void* dst, int R, int Cc, void* stream) {
    if (!src || !dst) return GLIDE_E_NULL;
    if (R < 1 || Cc < 1) return GLIDE_E_SHAPE;
    dim3 grid((Cc + 31) / 32, (R + 31) / 32);
    glide::count_launch(), glide::transpose_bf16_k<<<grid, dim3(32, 8), 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)src,
                                                                           (__nv_bfloat16*)dst, R, Cc);
    return (int)cudaGetLastError();
}

extern "C" int glide_pool2_bf16(const void* x, void* y, int Bn, int H, int W, int C, void* stream) {
    if (!x || !y) return GLIDE_E_NULL;
    if (Bn < 1 || H < 2 || W < 2 || H % 2 || W % 2 || C < 8 || C % 8) return GLIDE_E_SHAPE;
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) return GLIDE_E_SHAPE;
    const int64_t total = int64_t(Bn) * (H / 2) * (W / 2) * (C / 8);
    if ((total + 255) / 256 >= (int64_t(1) << 31)) return GLIDE_E_TOO_LARGE;
    glide::count_launch(), glide::pool2_k<<<unsigned((total + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
        (const uint4*)x, (uint4*)y, H / 2, W / 2, C / 8, total);
    return (int)cudaGetLastError();
}

extern "C" int glide_guess_features(int dtype, const void* H, const void* bed, const void* beta, const void* B, void* x,
                                    int64_t n, void* stream) {
    if (dtype != GLIDE_F32 && dtype != GLIDE_F64) return GLIDE_E_DTYPE;
    if (!H || !bed || !beta || !B || !x) return GLIDE_E_NULL;
    if (n < 1 || (reinterpret_cast<uintptr_t>(x) & 15)) return GLIDE_E_SHAPE;
    if ((n + 255) / 256 >= (int64_t(1) << 31)) return GLIDE_E_TOO_LARGE;
    const unsigned nb = unsigned((n + 255) / 256);
    glide::count_launch();
    if (dtype == GLIDE_F32)
        glide::guess_features_k<float><<<nb, 256, 0, (cudaStream_t)stream>>>(
            (const float*)H, (const float*)bed, (const float*)beta, (const float*)B, (uint4*)x, n);
    else
        glide::guess_features_k<double><<<nb, 256, 0, (cudaStream_t)stream>>>(
            (const double*)H, (const double*)bed, (const double*)beta, (const double*)B, (uint4*)x, n);
    return (int)cudaGetLastError();
}

extern "C" int glide_guess_faces(const float* pred, double* u, double* v, int nb, int ny, int nx, double scale,
                                 void* stream) {
    if (!pred || !u || !v) return GLIDE_E_NULL;
    if (nb < 1 || nb > 65535 || ny < 1 || nx < 1 || (reinterpret_cast<uintptr_t>(pred) & 7)) return GLIDE_E_SHAPE;
    const dim3 grid((nx + 1 + 31) / 32, (ny + 1 + 7) / 8, nb);
    if (grid.y > 65535) return GLIDE_E_TOO_LARGE;
    glide::count_launch(), glide::guess_faces_k<<<grid, dim3(32, 8), 0, (cudaStream_t)stream>>>(
        (const float2*)pred, u, v, ny, nx, float(scale));
    return (int)cudaGetLastError();
}
