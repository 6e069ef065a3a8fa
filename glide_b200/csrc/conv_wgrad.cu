// Backward pieces of a 3x3 layer of the learned guess on the tensor cores.
//
// Weight gradient  dW[co, tap*C + c] = sum_p gz[p, co] x[shift_tap(p), c]: the
// contraction runs over the pixels, which are the rows of both NHWC operands,
// so both are read MN-major as they lie in memory -- no im2col matrix, no
// transposes.  One CTA owns 32 input channels of one tap (and up to 128 output
// channels) and walks all pixels: a ring of 256-pixel stages, filled by tensor
// copies whose box is the tap's shifted rectangle (or, where 256 consecutive
// pixels are no rectangle, by copy warps that gather 16 bytes at a time), and
// one warp that issues sixteen K = 16 MMAs per stage.  The pixels are
// accumulated one after the other in FP32, in the order the GEMM on the
// explicit im2col matrix accumulates them, so the sums are the same bits; a
// split of the pixels over CTAs would change them.  What bounds it is that
// serial chain, 32,768 MMAs on eight 256^2 patches: 1.20 ms (70 clocks per MMA;
// stages of 128 pixels 1.52 ms, gathered 2.14 ms), where transposes and GEMM
// took 12.4 ms.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

#include "glide_b200.h"
#include "tc_common.cuh"

namespace glide {
void count_launch();

constexpr int WG_K = 256;                         // pixels per stage
constexpr int WG_BN = 32;                         // input channels per CTA
constexpr int WG_COPY = 256;                      // copy threads
constexpr int WG_THREADS = WG_COPY + 32;
constexpr int WG_MAXST = 7;
constexpr uint32_t WG_BLOCK = WG_K * 64;          // 32 channels x WG_K pixels, one 64-byte row per pixel
constexpr uint32_t WG_SMEM = 224 * 1024;

// 16 bytes of pixel row px, column c of four: permuted in groups of 8 rows (64-byte swizzle)
__device__ __forceinline__ uint32_t wg_off(int px, int c) { return uint32_t(px * 64 + ((c ^ ((px >> 1) & 3)) << 4)); }

struct ConvWgrad {
    const __nv_bfloat16 *gz, *x;
    float* dW;
    int Bn, H, Wd, C, N;   // N output channels, C input channels
    int ablocks, stages;   // 32-channel blocks of gz per stage; ring
    int bw, bh;            // TMA: a stage is bh image rows of bw pixels
    int* err;
};

__device__ __forceinline__ void tma_2d(uint32_t dst, const CUtensorMap* m, int c, int p, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            dst),
        "l"(m), "r"(c), "r"(p), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void tma_4d(uint32_t dst, const CUtensorMap* m, int c, int x, int y, int b, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];" ::"r"(dst),
        "l"(m), "r"(c), "r"(x), "r"(y), "r"(b), "r"(smem_u32(bar))
        : "memory");
}

// TMA: a stage's pixels are a rectangle of whole or partial image rows (the
// launcher checks), so one thread fetches it with two or five tensor copies
// (zero-filled outside the image); else the copy warps gather 16 bytes at a
// time.
template <bool TMA>
__global__ void __launch_bounds__(WG_THREADS) conv_wgrad_kernel(const ConvWgrad a, const __grid_constant__ CUtensorMap tg,
                                                                const __grid_constant__ CUtensorMap tx) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[WG_MAXST], empty[WG_MAXST], drain;
    __shared__ uint32_t tmem_slot;
    const int tid = threadIdx.x, warp = tid / 32, lane = tid & 31;
    const int tap = blockIdx.x % 9, c0 = (blockIdx.x / 9) * WG_BN, n0 = blockIdx.y * 128;
    const int dy = tap / 3 - 1, dx = tap % 3 - 1;
    const uint32_t base = (smem_u32(smem) + 1023u) & ~1023u;
    const int64_t P = int64_t(a.Bn) * a.H * a.Wd;
    const int n_st = int((P + WG_K - 1) / WG_K), S = a.stages;
    const uint32_t stage = uint32_t(a.ablocks + 1) * WG_BLOCK;
    if (warp == WG_COPY / 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(uint32_t(WG_BN)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    if (tid == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(&full[s], TMA ? 1 : WG_COPY);
            mbar_init(&empty[s], 1);
        }
        mbar_init(&drain, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // channels past N and C are never copied: they stay zero
    for (uint32_t k = tid; k < WG_SMEM / 16; k += WG_THREADS)
        asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(base + k * 16), "r"(0u) : "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    bool ok = true;

    if (TMA && warp < WG_COPY / 32) {
        if (tid == 0) {
            int sl = 0, x = 0, y = 0, b = 0, sent = 0;
            uint32_t turn = 1;
            for (int r = 0; r < n_st; r++) {
                if (r >= S && !mbar_wait_bounded(smem_u32(&empty[sl]), turn)) {
                    ok = false;
                    break;
                }
                const uint32_t st = base + uint32_t(sl) * stage;
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&full[sl])),
                             "r"(stage)
                             : "memory");
                for (int k = 0; k < a.ablocks; k++)
                    tma_2d(st + uint32_t(k) * WG_BLOCK, &tg, n0 + k * 32, r * WG_K, &full[sl]);
                tma_4d(st + uint32_t(a.ablocks) * WG_BLOCK, &tx, c0, x + dx, y + dy, b, &full[sl]);
                sent = r + 1;
                x += a.bw;
                if (x >= a.Wd) {
                    x = 0;
                    y += a.bh;
                    if (y >= a.H) {
                        y = 0;
                        b++;
                    }
                }
                if (++sl == S) {
                    sl = 0;
                    turn ^= 1;
                }
            }
            // every copy has landed before the CTA may end
            for (int r = sent > S ? sent - S : 0; r < sent; r++)
                if (!mbar_wait_bounded(smem_u32(&full[r % S]), uint32_t((r / S) & 1))) ok = false;
        }
        __syncwarp();
    } else if (warp < WG_COPY / 32) {
        // thread -> 16-byte column c of pixels tid / 4 + 64 h of a stage
        const int c = tid & 3;
        const int na = min(128, a.N - n0) - c * 8, nb = a.C - c0 - c * 8;   // channels left from this column on
        constexpr int NH = WG_K / 64;
        const __nv_bfloat16 *g[NH], *q[NH];
        int64_t left[NH];
        int xx[NH], yy[NH];
#pragma unroll
        for (int h = 0; h < NH; h++) {
            const int64_t p = (tid >> 2) + 64 * h;
            left[h] = P - p;
            xx[h] = int(p % a.Wd) + dx;
            yy[h] = int((p / a.Wd) % a.H) + dy;
            g[h] = a.gz + p * a.N + n0 + c * 8;
            q[h] = a.x + (p + int64_t(dy) * a.Wd + dx) * a.C + c0 + c * 8;
        }
        const uint32_t o0 = wg_off(tid >> 2, c), ob = uint32_t(a.ablocks) * WG_BLOCK;
        int sl = 0;
        uint32_t turn = 1;   // parity of the stage's previous release
        for (int r = 0; r < n_st; r++) {
            if (r >= S && !mbar_wait_bounded(smem_u32(&empty[sl]), turn)) {
                ok = false;
                break;
            }
#pragma unroll
            for (int h = 0; h < NH; h++) {
                const uint32_t st = base + uint32_t(sl) * stage + o0 + uint32_t(h) * (64 * 64);
                const bool in = left[h] > 0;
                for (int k = 0; k * 32 < na; k++)
                    cp_async16(st + uint32_t(k) * WG_BLOCK, in ? g[h] + k * 32 : a.gz, in ? 16u : 0u);
                const bool xin = in && unsigned(yy[h]) < unsigned(a.H) && unsigned(xx[h]) < unsigned(a.Wd);
                if (nb > 0) cp_async16(st + ob, xin ? q[h] : a.x, xin ? 16u : 0u);
                left[h] -= WG_K;
                g[h] += WG_K * a.N;
                q[h] += WG_K * a.C;
                xx[h] += WG_K;
                while (xx[h] - dx >= a.Wd) {
                    xx[h] -= a.Wd;
                    if (++yy[h] - dy == a.H) yy[h] = dy;
                }
            }
            cp_async_arrive(&full[sl]);
            if (++sl == S) {
                sl = 0;
                turn ^= 1;
            }
        }
        cp_async_commit();
        cp_async_wait<0>();
    } else {
        const uint32_t idesc = idesc_bf16_f32(128, WG_BN, true), lead = lane == 0, hi = umma_hi_mn_sw64();
        // with one block of output channels the tile's other rows read it again (they are not stored)
        const uint32_t a_step = a.ablocks > 1 ? WG_BLOCK : 0;
        int sl = 0;
        uint32_t turn = 0;
        for (int r = 0; r < n_st; r++) {
            if (!mbar_wait_bounded(smem_u32(&full[sl]), turn)) { ok = false; break; }
            if (TMA)
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            else
                fence_copied();
            const uint32_t st = base + uint32_t(sl) * stage;
            const uint32_t a_lo = umma_lo(st, a_step), b_lo = umma_lo(st + uint32_t(a.ablocks) * WG_BLOCK, WG_BLOCK);
#pragma unroll
            for (int k = 0; k < WG_K / 16; k++)   // 16 pixels: 1024 B
                mma_bf16_lead(tmem, a_lo + k * 64, hi, b_lo + k * 64, hi, idesc, r > 0 || k > 0, lead);
            mma_commit_lead(&empty[sl], lead);
            if (++sl == S) {
                sl = 0;
                turn ^= 1;
            }
        }
        mma_commit_lead(&drain, lead);
        if (!mbar_wait_bounded(smem_u32(&drain), 0)) ok = false;
    }
    if (!ok && lane == 0 && a.err) atomicExch(a.err, 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp < 4) {
        float v[WG_BN];
        tmem_load<WG_BN>(tmem + (uint32_t(warp * 32) << 16), v);
        const int n = n0 + warp * 32 + lane;
        if (n < a.N) {
            float* o = a.dW + int64_t(n) * 9 * a.C + int64_t(tap) * a.C + c0;
#pragma unroll
            for (int e = 0; e < WG_BN; e++)
                if (c0 + e < a.C) o[e] = v[e];
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == WG_COPY / 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(uint32_t(WG_BN)));
}

// gz = gy where y > 0 (all of gy without relu), per-block channel sums of gz.
// Thread layout: N / 8 threads along the channels, the rest along the pixels.
constexpr int RG_NT = 256;
__global__ void __launch_bounds__(RG_NT) relu_grad_kernel(const __nv_bfloat16* __restrict__ gy,
                                                          const __nv_bfloat16* __restrict__ y,
                                                          __nv_bfloat16* __restrict__ gz, float* __restrict__ parts,
                                                          int64_t P, int N, int relu) {
    extern __shared__ float sh[];   // rows x N
    const int nch = N / 8, rows = RG_NT / nch;
    const int ch = threadIdx.x % nch, pr = threadIdx.x / nch;
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (pr < rows) {
        for (int64_t p = int64_t(blockIdx.x) * rows + pr; p < P; p += int64_t(gridDim.x) * rows) {
            const int64_t o = p * N + ch * 8;
            uint4 gv = *reinterpret_cast<const uint4*>(gy + o);
            __nv_bfloat16* gh = reinterpret_cast<__nv_bfloat16*>(&gv);
            if (relu) {
                const uint4 yv = *reinterpret_cast<const uint4*>(y + o);
                const __nv_bfloat16* yh = reinterpret_cast<const __nv_bfloat16*>(&yv);
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    const float m = __bfloat162float(yh[e]) > 0.0f ? 1.0f : 0.0f;
                    gh[e] = __float2bfloat16(__bfloat162float(gh[e]) * m);
                }
            }
            *reinterpret_cast<uint4*>(gz + o) = gv;
#pragma unroll
            for (int e = 0; e < 8; e++) acc[e] += __bfloat162float(gh[e]);
        }
#pragma unroll
        for (int e = 0; e < 8; e++) sh[pr * N + ch * 8 + e] = acc[e];
    }
    __syncthreads();
    for (int n = threadIdx.x; n < N; n += RG_NT) {
        float s = 0.0f;
        for (int r = 0; r < rows; r++) s += sh[r * N + n];
        parts[int64_t(blockIdx.x) * N + n] = s;
    }
}
// db[n] = sum of the blocks' sums, in block order, FP64
__global__ void relu_grad_sum_kernel(const float* __restrict__ parts, float* __restrict__ db, int nblk, int N) {
    const int n = blockIdx.x, lane = threadIdx.x;
    double s = 0.0;
    for (int k = lane; k < nblk; k += 32) s += double(parts[int64_t(k) * N + n]);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) db[n] = float(s);
}

}  // namespace glide

namespace {
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encode_tiled() {
    static EncodeTiled fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiled>(f);
    });
    return fn;
}

// BF16 NHWC tensor in boxes of 32 channels, 64-byte swizzle
bool tensor_map(CUtensorMap* m, const void* base, int rank, const cuuint64_t* dims, const cuuint32_t* box) {
    EncodeTiled enc = encode_tiled();
    if (!enc) return false;
    cuuint64_t strides[4];
    cuuint64_t s = dims[0] * 2;
    for (int k = 0; k + 1 < rank; k++) {
        strides[k] = s;
        s *= dims[k + 1];
    }
    const cuuint32_t one[4] = {1, 1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, cuuint32_t(rank), const_cast<void*>(base), dims, strides, box, one,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <bool TMA>
int launch_wgrad(const glide::ConvWgrad& a, const CUtensorMap& tg, const CUtensorMap& tx, cudaStream_t s) {
    using namespace glide;
    constexpr int SMEM = WG_SMEM + 1024;
    static int configured[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return GLIDE_E_SHAPE;
    if (!configured[dev]) {
        const cudaError_t e =
            cudaFuncSetAttribute(conv_wgrad_kernel<TMA>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (e != cudaSuccess) return int(e);
        configured[dev] = 1;
    }
    const dim3 grid(9 * ((a.C + WG_BN - 1) / WG_BN), (a.N + 127) / 128);
    count_launch(), conv_wgrad_kernel<TMA><<<grid, WG_THREADS, SMEM, s>>>(a, tg, tx);
    return int(cudaGetLastError());
}
}  // namespace

extern "C" int glide_conv3x3_wgrad_bf16(const void* gz, const void* x, float* dW, int Bn, int H, int W, int C, int N,
                                        int* err, void* stream) {
    using namespace glide;
    if (!gz || !x || !dW) return GLIDE_E_NULL;
    if (Bn < 1 || H < 1 || W < 1 || C < 8 || C % 8 || N < 8 || N % 8) return GLIDE_E_SHAPE;
    if (((reinterpret_cast<uintptr_t>(gz) | reinterpret_cast<uintptr_t>(x)) & 15)) return GLIDE_E_SHAPE;
    if (int64_t(Bn) * H * W >= (int64_t(1) << 31)) return GLIDE_E_TOO_LARGE;
    ConvWgrad a{(const __nv_bfloat16*)gz, (const __nv_bfloat16*)x, dW, Bn, H, W, C, N, 0, 0, 0, 0, err};
    // a tile of 128 rows reads one or four blocks
    a.ablocks = N <= 32 ? 1 : 4;
    const int st = int(WG_SMEM / ((a.ablocks + 1) * WG_BLOCK));
    a.stages = st < WG_MAXST ? st : WG_MAXST;
    CUtensorMap tg{}, tx{};
    // the pixels of a stage are a rectangle when rows hold a multiple of WG_K pixels or divide it evenly
    a.bw = W < WG_K ? W : WG_K;
    a.bh = WG_K / a.bw;
    if (W % a.bw == 0 && a.bw * a.bh == WG_K && H % a.bh == 0) {
        const cuuint64_t dg[2] = {cuuint64_t(N), cuuint64_t(Bn) * H * W};
        const cuuint32_t bg[2] = {32, WG_K};
        const cuuint64_t dx[4] = {cuuint64_t(C), cuuint64_t(W), cuuint64_t(H), cuuint64_t(Bn)};
        const cuuint32_t bx[4] = {32, cuuint32_t(a.bw), cuuint32_t(a.bh), 1};
        if (tensor_map(&tg, gz, 2, dg, bg) && tensor_map(&tx, x, 4, dx, bx))
            return launch_wgrad<true>(a, tg, tx, (cudaStream_t)stream);
    }
    return launch_wgrad<false>(a, tg, tx, (cudaStream_t)stream);
}

extern "C" int glide_relu_grad_blocks(int64_t P, int N) {
    const int64_t rows = glide::RG_NT / (N / 8 > 0 ? N / 8 : 1);
    int64_t b = rows > 0 ? (P + rows * 8 - 1) / (rows * 8) : 1;
    return int(b > 592 ? 592 : (b < 1 ? 1 : b));
}

extern "C" int glide_relu_grad_bf16(const void* gy, const void* y, void* gz, float* db, float* parts, int64_t P,
                                    int N, int relu, void* stream) {
    using namespace glide;
    if (!gy || !gz || !db || !parts || (relu && !y)) return GLIDE_E_NULL;
    if (P < 1 || N < 8 || N % 8 || N / 8 > RG_NT) return GLIDE_E_SHAPE;
    if (((reinterpret_cast<uintptr_t>(gy) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(gz)) & 15))
        return GLIDE_E_SHAPE;
    const int nb = glide_relu_grad_blocks(P, N);
    const size_t sm = size_t(RG_NT / (N / 8)) * N * sizeof(float);
    count_launch(), relu_grad_kernel<<<nb, RG_NT, sm, (cudaStream_t)stream>>>(
        (const __nv_bfloat16*)gy, (const __nv_bfloat16*)y, (__nv_bfloat16*)gz, parts, P, N, relu);
    count_launch(), relu_grad_sum_kernel<<<N, 32, 0, (cudaStream_t)stream>>>(parts, db, nb, N);
    return int(cudaGetLastError());
}
