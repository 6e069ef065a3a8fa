// 3x3 convolution of the learned guess as a march down image rows on the
// 5th-generation tensor cores.
//
//   out[p, n] = act(bias[n] + sum_{ky,kx,c} x[y+ky-1, x+kx-1, c] W[n, (ky*3+kx)*C + c])
//
// What bounds it: the issue of narrow MMAs and, per row, the copy -> product ->
// store latency that the ring and the resident CTAs have to cover.  1024^2,
// 32 -> 32: 226 us as an implicit GEMM, 52 us here (134 MB, 2.6 TB/s); 512^2,
// 64 -> 64: 163 -> 37.
//
// The implicit GEMM of tc_gemm.cu gathers nine shifted copies of its 128
// pixels (73 KB of copies for 8 KB of input at C = 32) and runs load, product
// and store of a CTA one after the other; at 1024^2 and C = 32 it held the
// tensor pipe 3 % active.  Here a CTA owns 128 columns (and up to 64 output
// channels) of an image and streams the input rows of a chunk through a ring
// of shared-memory stages, each row copied once: a row is kept as planes of 8
// channels with one 16-byte entry per pixel, so a tap's shift by one pixel is
// a shift of the operand's start address by 16 bytes, and the nine taps of a
// 128-pixel tile are nine views of three rows.  Input row j feeds the output
// rows j+1, j and j-1 (ky = 0, 1, 2), whose FP32 accumulators live in a
// four-row ring of TMEM; a row's products are issued in the order ky, kx, c,
// as the implicit GEMM issues them, so the results are the same bits.  Warps
// are specialised: four copy rows (cp.async, zero-filled outside the image),
// two issue the MMAs, four drain finished accumulators (bias, ReLU, BF16 or
// FP32 stores), so copies, products and stores of different rows overlap.  The
// two MMA warps take the even and the odd output rows: one warp's issue (a
// narrow MMA every 90 clocks, 40 needed) does not keep the pipe busy at 96
// channels and more, where one CTA fits an SM (1024^2, 96 -> 32: 127 us with
// one, 105 with two; 512^2, 192 -> 64: 136 -> 122; others within 3 %).  The input may be the channel concatenation of two tensors, the
// first at half resolution (nearest upsampling): the copy warps read both
// sources directly and neither the upsampled nor the joined tensor exists.
//
// C = 8 (the network's input layer) stages, per output row, the nine shifted
// pixel planes themselves (K = 72, padded to 80 by a plane of zeros).
//
// Every wait is bounded: a role whose wait runs out (~1 s) sets *err = 1 and
// leaves its loop; the others run out likewise, the MMAs in flight are waited
// for (bounded), TMEM is freed and the kernel returns.
#include <cuda_bf16.h>
#include <stdint.h>

#include "glide_b200.h"
#include "tc_common.cuh"

namespace glide {
void count_launch();

constexpr int CR_PX = 130;                       // staged pixels of a row: 128 + one each side
constexpr int CR_ROLE = 128;                     // copy threads = store threads
constexpr int CR_MMA = 2;                        // MMA warps, one per parity of the output row
constexpr int CR_THREADS = 2 * CR_ROLE + 32 * CR_MMA;
constexpr int CR_ACC = 4;                        // accumulator rows in flight
constexpr int CR_MAXST = 8;
constexpr uint32_t CR_PLANE = CR_PX * 16;        // bytes of one 8-channel plane of a staged row
constexpr uint32_t CR_PLANE8 = 128 * 16;         // C = 8: one tap's plane
constexpr int CR_PLANES8 = 10;                   // 9 taps + zeros
constexpr size_t CR_SMEM_MAX = 225 * 1024;       // dynamic shared memory of one CTA
constexpr size_t CR_SMEM_SM = 227 * 1024;        // of one SM

struct ConvRows {
    const __nv_bfloat16 *x0, *x1;   // x1: channels C0.. at full resolution (null without a second source)
    int C0, C1, up0;                // up0: x0 is (H/2, W/2), read at (y/2, x/2)
    const void* W;                  // BF16, or FP32 (rounded to BF16 while it is staged)
    int ldw, w32;
    void* out;
    int ldc, N;
    const float* bias;
    int relu, out_mode;             // 0: FP32, 1: BF16
    int* err;
    int Bn, H, Wd, strips, rows, chunks, stages;
};

// KS: K steps per tap (C / 16) when known at compile time, else 0
template <int BN, bool C8, int KS>
__global__ void __launch_bounds__(CR_THREADS) conv_rows_kernel(const ConvRows a) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[CR_MAXST], empty[CR_MAXST], acc_full[CR_ACC], acc_empty[CR_ACC], drain[CR_MMA];
    __shared__ uint32_t tmem_slot;
    const int tid = threadIdx.x, warp = tid / 32, lane = tid & 31;
    const int C = a.C0 + a.C1, S = a.stages;
    const int strip = blockIdx.x % a.strips, t = blockIdx.x / a.strips;
    const int chunk = t % a.chunks, img = t / a.chunks;
    const int n0 = blockIdx.y * BN;
    const int xs = strip * 128;
    const int y0 = chunk * a.rows, y1 = min(y0 + a.rows, a.H);
    const int n_in = C8 ? y1 - y0 : y1 - y0 + 2;           // staged rows
    const int kplanes = C8 ? CR_PLANES8 : 9 * C / 8;
    const uint32_t sB = (smem_u32(smem) + 127u) & ~127u;
    const uint32_t sA = sB + uint32_t(kplanes) * BN * 16;
    const uint32_t stage_bytes = C8 ? CR_PLANES8 * CR_PLANE8 : uint32_t(C / 8) * CR_PLANE;

    if (warp == 8) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(uint32_t(CR_ACC * BN)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    if (tid == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(&full[s], CR_ROLE);
            mbar_init(&empty[s], CR_MMA);
        }
        for (int s = 0; s < CR_ACC; s++) {
            mbar_init(&acc_full[s], 1);
            mbar_init(&acc_empty[s], 4);
        }
        for (int s = 0; s < CR_MMA; s++) mbar_init(&drain[s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // weights: plane k/8, row n, 16 bytes
    for (int k = tid; k < kplanes * BN; k += CR_THREADS) {
        const int pl = k / BN, n = k - pl * BN;
        const bool ok = n0 + n < a.N && pl * 8 < 9 * C;
        const int64_t o = ok ? int64_t(n0 + n) * a.ldw + pl * 8 : 0;
        if (a.w32) {
            const float4* q = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(a.W) + o);
            const float4 lo = ok ? __ldg(q) : make_float4(0, 0, 0, 0), hi = ok ? __ldg(q + 1) : make_float4(0, 0, 0, 0);
            const __nv_bfloat162 h[4] = {__floats2bfloat162_rn(lo.x, lo.y), __floats2bfloat162_rn(lo.z, lo.w),
                                         __floats2bfloat162_rn(hi.x, hi.y), __floats2bfloat162_rn(hi.z, hi.w)};
            const uint32_t* w = reinterpret_cast<const uint32_t*>(h);
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sB + uint32_t(k) * 16), "r"(w[0]), "r"(w[1]),
                         "r"(w[2]), "r"(w[3])
                         : "memory");
        } else {
            cp_async16(sB + uint32_t(k) * 16, reinterpret_cast<const __nv_bfloat16*>(a.W) + o, ok ? 16u : 0u);
        }
    }
    if (C8)
        for (int k = tid; k < S * 128; k += CR_THREADS)
            cp_async16(sA + uint32_t(k / 128) * stage_bytes + 9 * CR_PLANE8 + uint32_t(k % 128) * 16, a.W, 0u);
    cp_async_commit();
    cp_async_wait<0>();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    bool ok = true;

    if (warp < 4) {
        // ---------------------------------------------------------------- copy rows
        const int c8 = C / 8, c08 = a.C0 / 8;
        const int items = C8 ? 9 * 128 : CR_PX * c8;
        auto copy_row = [&](int r) {
            const uint32_t st = sA + uint32_t(r % S) * stage_bytes;
            if constexpr (C8) {
                const int y = y0 + r;
                for (int k = tid; k < items; k += CR_ROLE) {
                    const int tap = k / 128, m = k & 127;
                    const int ky = tap / 3, kx = tap - 3 * ky;
                    const int sy = y + ky - 1, sx = xs + m + kx - 1;
                    const bool in = sy >= 0 && sy < a.H && sx >= 0 && sx < a.Wd && xs + m < a.Wd;
                    cp_async16(st + uint32_t(k) * 16,
                               in ? a.x0 + ((int64_t(img) * a.H + sy) * a.Wd + sx) * 8 : a.x0, in ? 16u : 0u);
                }
            } else {
                const int sy = y0 - 1 + r;
                const bool yin = sy >= 0 && sy < a.H;
                const int yy = yin ? sy : 0;
                const __nv_bfloat16* r0 =
                    a.up0 ? a.x0 + (int64_t(img) * (a.H / 2) + yy / 2) * (a.Wd / 2) * a.C0
                          : a.x0 + (int64_t(img) * a.H + yy) * a.Wd * a.C0;
                const __nv_bfloat16* r1 = a.x1 ? a.x1 + (int64_t(img) * a.H + yy) * a.Wd * a.C1 : nullptr;
                int px = tid / c8, c = tid - px * c8;
                const int dpx = CR_ROLE / c8, dc = CR_ROLE - dpx * c8;
                for (int k = tid; k < items; k += CR_ROLE) {
                    const int sx = xs - 1 + px;
                    const bool in = yin && sx >= 0 && sx < a.Wd;
                    const __nv_bfloat16* src =
                        c < c08 ? r0 + ((a.up0 ? sx >> 1 : sx) * a.C0 + c * 8) : r1 + (sx * a.C1 + (c - c08) * 8);
                    cp_async16(st + uint32_t(c) * CR_PLANE + uint32_t(px) * 16, in ? src : a.x0, in ? 16u : 0u);
                    px += dpx;
                    c += dc;
                    if (c >= c8) { c -= c8; px++; }
                }
            }
        };
        for (int r = 0; r < n_in; r++) {
            if (r >= S && !mbar_wait_bounded(smem_u32(&empty[r % S]), uint32_t((r / S - 1) & 1))) {
                ok = false;
                break;
            }
            copy_row(r);
            cp_async_arrive(&full[r % S]);
        }
        cp_async_commit();
        cp_async_wait<0>();
    } else if (warp >= 8) {
        // ---------------------------------------------------------------- products (the whole warp, lane 0 issues)
        const int me = warp - 8;
        const uint32_t idesc = idesc_bf16_f32(128, BN), lead = lane == 0;
        const uint32_t a_hi = umma_hi(128), b_hi = umma_hi(128);
        for (int r = 0; r < n_in && ok; r++) {
            if (!mbar_wait_bounded(smem_u32(&full[r % S]), uint32_t((r / S) & 1))) { ok = false; break; }
            fence_copied();
            const uint32_t st = sA + uint32_t(r % S) * stage_bytes;
            if constexpr (C8) {
                const int slot = r % CR_ACC;
                if ((r & 1) != me) {   // the other warp's row
                    mma_commit_lead(&empty[r % S], lead);
                    continue;
                }
                if (r >= CR_ACC && !mbar_wait_bounded(smem_u32(&acc_empty[slot]), uint32_t((r / CR_ACC - 1) & 1))) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a0 = umma_lo(st, CR_PLANE8), b0 = umma_lo(sB, BN * 16);
#pragma unroll
                for (int s = 0; s < CR_PLANES8 / 2; s++)
                    mma_bf16_lead(tmem + slot * BN, a0 + s * (2 * CR_PLANE8 / 16), a_hi, b0 + s * (2 * BN), b_hi, idesc,
                                  s > 0, lead);
                mma_commit_lead(&acc_full[slot], lead);
            } else {
                // ky = 2 finishes output row r-2 of the chunk, ky = 1 continues r-1, ky = 0 opens r
                const uint32_t a0 = umma_lo(st, CR_PLANE), b0 = umma_lo(sB, BN * 16);
                const int ks = KS ? KS : C / 16;
#pragma unroll
                for (int ky = 2; ky >= 0; ky--) {
                    const int yo = r - ky;
                    if (yo < 0 || yo >= y1 - y0 || (yo & 1) != me) continue;
                    const int slot = yo % CR_ACC;
                    if (ky == 0 && yo >= CR_ACC) {
                        if (!mbar_wait_bounded(smem_u32(&acc_empty[slot]), uint32_t((yo / CR_ACC - 1) & 1))) {
                            ok = false;
                            break;
                        }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    }
#pragma unroll
                    for (int kx = 0; kx < 3; kx++) {
#pragma unroll
                        for (int s = 0; s < ks; s++)
                            mma_bf16_lead(tmem + slot * BN, a0 + kx + s * (2 * CR_PLANE / 16), a_hi,
                                          b0 + ((ky * 3 + kx) * ks + s) * (2 * BN), b_hi, idesc,
                                          ky > 0 || kx > 0 || s > 0, lead);
                    }
                    if (ky == 2) mma_commit_lead(&acc_full[slot], lead);
                }
            }
            mma_commit_lead(&empty[r % S], lead);
        }
        // the MMAs in flight read shared memory: they end before the CTA does
        mma_commit_lead(&drain[me], lead);
        if (!mbar_wait_bounded(smem_u32(&drain[me]), 0)) ok = false;
        __syncwarp();
    } else {
        // ---------------------------------------------------------------- store finished rows
        const int w = warp - 4, m = w * 32 + lane, x = xs + m;
        const bool vec = (a.ldc & 7) == 0 && (reinterpret_cast<uintptr_t>(a.out) & 15) == 0;
        float bias[BN];
#pragma unroll
        for (int e = 0; e < BN; e++) bias[e] = a.bias && n0 + e < a.N ? __ldg(a.bias + n0 + e) : 0.0f;
        for (int yo = 0; yo < y1 - y0; yo++) {
            const int slot = yo % CR_ACC;
            if (!mbar_wait_bounded(smem_u32(&acc_full[slot]), uint32_t((yo / CR_ACC) & 1))) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float v[BN];
            tmem_load<BN>(tmem + (uint32_t(w * 32) << 16) + uint32_t(slot * BN), v);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[slot]);
            if (x >= a.Wd) continue;
            const int64_t o = ((int64_t(img) * a.H + y0 + yo) * a.Wd + x) * a.ldc + n0;
#pragma unroll
            for (int e = 0; e < BN; e++) {
                if (a.bias) v[e] += bias[e];
                if (a.relu) v[e] = fmaxf(v[e], 0.0f);
            }
#pragma unroll
            for (int c = 0; c < BN; c += 8) {
                if (n0 + c >= a.N) break;
                if (vec && n0 + c + 8 <= a.N) {
                    if (a.out_mode == 1) {
                        __align__(16) __nv_bfloat16 h[8];
#pragma unroll
                        for (int e = 0; e < 8; e++) h[e] = __float2bfloat16(v[c + e]);
                        *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(a.out) + o + c) =
                            *reinterpret_cast<uint4*>(h);
                    } else {
                        float4* q = reinterpret_cast<float4*>(reinterpret_cast<float*>(a.out) + o + c);
                        q[0] = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
                        q[1] = make_float4(v[c + 4], v[c + 5], v[c + 6], v[c + 7]);
                    }
                    continue;
                }
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    if (n0 + c + e >= a.N) break;
                    if (a.out_mode == 1) reinterpret_cast<__nv_bfloat16*>(a.out)[o + c + e] = __float2bfloat16(v[c + e]);
                    else reinterpret_cast<float*>(a.out)[o + c + e] = v[c + e];
                }
            }
        }
    }
    if (!ok && lane == 0 && a.err) atomicExch(a.err, 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 8)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(uint32_t(CR_ACC * BN)));
}

template <int BN, bool C8, int KS> int launch_conv_rows(const ConvRows& a, size_t smem, cudaStream_t s) {
    static int configured[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return GLIDE_E_SHAPE;
    if (!configured[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(conv_rows_kernel<BN, C8, KS>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, CR_SMEM_MAX);
        if (e != cudaSuccess) return int(e);
        configured[dev] = 1;
    }
    const dim3 grid(unsigned(a.strips) * a.chunks * a.Bn, (a.N + BN - 1) / BN);
    count_launch(), conv_rows_kernel<BN, C8, KS><<<grid, CR_THREADS, smem, s>>>(a);
    return int(cudaGetLastError());
}

// The narrow widths of the guess network have their K loop unrolled: with
// every descriptor an immediate away from two bases the issuing warp comes
// closer to the tensor pipe (about 90 clocks per MMA in a rolled loop, 40
// needed; 1024^2, 96 -> 32 with one MMA warp: 160 -> 129 us).  At 192 channels the unrolled body
// is slower than the loop (512^2, 192 -> 64: 180 against 138 us).
template <int BN> int pick_conv_rows(const ConvRows& a, bool c8, size_t smem, cudaStream_t s) {
    if (c8) return launch_conv_rows<BN, true, 0>(a, smem, s);
    switch (a.C0 + a.C1) {
        case 32: return launch_conv_rows<BN, false, 2>(a, smem, s);
        case 64: return launch_conv_rows<BN, false, 4>(a, smem, s);
        case 96: return launch_conv_rows<BN, false, 6>(a, smem, s);
        case 128: return launch_conv_rows<BN, false, 8>(a, smem, s);
        default: return launch_conv_rows<BN, false, 0>(a, smem, s);
    }
}

// The shapes of the row march: C = 8 (one source) or C a multiple of 16, the
// weights of 32 output channels and two staged rows within one SM's shared
// memory (C <= 224), and at least 64 columns, half of a tile's pixels.
bool conv_rows_takes(int C0, int up0, int C1, int W, int N) {
    const int C = C0 + C1;
    const bool c8 = C == 8 && !C1 && !up0;
    if (!(c8 || C % 16 == 0) || W < 64 || N < 1) return false;
    const size_t stage = c8 ? CR_PLANES8 * CR_PLANE8 : size_t(C / 8) * CR_PLANE;
    return size_t(c8 ? CR_PLANES8 : 9 * C / 8) * 32 * 16 + 128 + 2 * stage <= CR_SMEM_MAX;
}

// Launches the row march and returns its status, or returns -1000 where the
// call is not one of its own: another shape, out_mode 2, operands that are not
// 16-byte aligned.
int try_conv_rows(const void* x0, int C0, int up0, const void* x1, int C1, int Bn, int H, int W, const void* Wt,
                  int ldw, int w32, void* out, int ldc, int N, const float* bias, int relu, int out_mode, int* err,
                  cudaStream_t s) {
    if (!conv_rows_takes(C0, up0, C1, W, N) || out_mode > 1 || ldw % 8 != 0) return -1000;
    const int C = C0 + C1;
    const bool c8 = C == 8;
    if (((reinterpret_cast<uintptr_t>(x0) | reinterpret_cast<uintptr_t>(x1) | reinterpret_cast<uintptr_t>(Wt)) & 15))
        return -1000;
    ConvRows a{};
    a.x0 = (const __nv_bfloat16*)x0; a.x1 = (const __nv_bfloat16*)x1;
    a.C0 = C0; a.C1 = C1; a.up0 = up0;
    a.W = Wt; a.ldw = ldw; a.w32 = w32;
    a.out = out; a.ldc = ldc; a.N = N; a.bias = bias; a.relu = relu; a.out_mode = out_mode; a.err = err;
    a.Bn = Bn; a.H = H; a.Wd = W;
    a.strips = (W + 127) / 128;
    const size_t stage = c8 ? CR_PLANES8 * CR_PLANE8 : size_t(C / 8) * CR_PLANE;
    const int kplanes = c8 ? CR_PLANES8 : 9 * C / 8;
    auto weights = [&](int bn) { return size_t(kplanes) * bn * 16 + 128; };
    const int bn = N > 32 && weights(64) + 2 * stage <= CR_SMEM_MAX ? 64 : 32;
    // as many CTAs per SM as shared memory and TMEM leave at least four stages each (or the one
    // that fits); registers hold two of 32 channels or one of 64 at a time, which is what an image
    // of few rows should be cut for: more CTAs would be a second wave of single rows, each staging
    // three (eight 64^2 images, 16 -> 32: 18.4 us, 9.1 with two per SM; before the march 14.3)
    const int64_t total = int64_t(Bn) * a.strips * H * ((N + bn - 1) / bn);
    const int most = 512 / (CR_ACC * bn);
    int occ = 1;
    for (int o = total < 4 * 148 * most ? most / 2 : most; o > 1; o--)
        if (weights(bn) + 4 * stage + 1024 <= CR_SMEM_SM / o) {
            occ = o;
            break;
        }
    const size_t room = occ > 1 ? CR_SMEM_SM / occ - 1024 : CR_SMEM_MAX;
    int64_t st = int64_t((room - weights(bn)) / stage);
    a.stages = int(st < CR_MAXST ? st : CR_MAXST);
    int64_t rows = (total + 148 * occ - 1) / (148 * occ);
    a.rows = int(rows < H ? rows : H);
    a.chunks = (H + a.rows - 1) / a.rows;
    const size_t smem = weights(bn) + a.stages * stage;
    return bn == 64 ? pick_conv_rows<64>(a, c8, smem, s) : pick_conv_rows<32>(a, c8, smem, s);
}

}  // namespace glide

extern "C" int glide_conv3x3_rows_ok(int C0, int up0, int C1, int W, int N) {
    return C0 >= 8 && C1 >= 0 && C0 % 8 == 0 && C1 % 8 == 0 && glide::conv_rows_takes(C0, up0, C1, W, N) ? 1 : 0;
}

extern "C" int glide_conv3x3_rows_f32w(const void* x0, int C0, int up0, const void* x1, int C1, int Bn, int H, int W,
                                       const float* Wt, void* out, int N, const float* bias, int relu, int* err,
                                       void* stream) {
    if (!x0 || !Wt || !out || (C1 > 0) != (x1 != nullptr)) return GLIDE_E_NULL;
    if (Bn < 1 || H < 1 || W < 1 || !glide_conv3x3_rows_ok(C0, up0, C1, W, N) || (up0 && (H % 2 || W % 2)))
        return GLIDE_E_SHAPE;
    if (int64_t(Bn) * H * W >= (int64_t(1) << 31)) return GLIDE_E_TOO_LARGE;
    const int rc = glide::try_conv_rows(x0, C0, up0, x1, C1, Bn, H, W, Wt, 9 * (C0 + C1), 1, out, N, N, bias, relu, 1,
                                        err, (cudaStream_t)stream);
    return rc == -1000 ? GLIDE_E_SHAPE : rc;
}
