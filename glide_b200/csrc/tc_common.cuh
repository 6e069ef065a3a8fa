// Shared pieces of the tcgen05 kernels: descriptors, mbarriers with bounded
// waits, cp.async, MMA issue and TMEM loads.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

namespace glide {

constexpr long long WAIT_CYCLES = 2000000000LL;  // ~1 s at 2 GHz

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// UMMA shared-memory matrix descriptor, no swizzle (SM100 version 1).
// K-major operands: lbo = the two 8-column halves of a K step, sbo = groups of
// 8 rows.  MN-major operands: lbo = groups of 8 along K, sbo = groups of 8
// along M/N.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= uint64_t((saddr >> 4) & 0x3FFFu);
    d |= uint64_t((lbo_bytes >> 4) & 0x3FFFu) << 16;
    d |= uint64_t((sbo_bytes >> 4) & 0x3FFFu) << 32;
    d |= uint64_t(1) << 46;
    return d;
}

// Instruction descriptor: D = F32, A = B = BF16, M x N; mn: both operands MN-major.
__host__ __device__ constexpr uint32_t idesc_bf16_f32(int M, int N, bool mn = false) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (mn ? (1u << 15) | (1u << 16) : 0u) | (uint32_t(N >> 3) << 17) |
           (uint32_t(M >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t da, uint64_t db, uint32_t idesc, bool acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
        :
        : "r"(tmem), "l"(da), "l"(db), "r"(idesc), "r"(acc ? 1u : 0u), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
        : "memory");
}

// The same with the descriptors as a start word (address and leading offset,
// which steps of an operand change by a constant) and a fixed upper word, issued by
// the lane whose `lead` is set: the loops around it are run by the whole warp,
// so their arithmetic stays uniform.
__device__ __forceinline__ uint32_t umma_lo(uint32_t saddr, uint32_t lbo_bytes) {
    return ((saddr >> 4) & 0x3FFFu) | (((lbo_bytes >> 4) & 0x3FFFu) << 16);
}
__device__ __forceinline__ uint32_t umma_hi(uint32_t sbo_bytes) { return ((sbo_bytes >> 4) & 0x3FFFu) | (1u << 14); }
// K-major operand of 64 columns in 128-byte rows whose 16-byte entries are
// permuted (entry ^ row % 8) within groups of 8 rows (1024-byte aligned): a row
// is one shared-memory line, so cp.async copies of it stay coalesced; a K step
// of 16 is 32 bytes.
__device__ __forceinline__ uint32_t umma_hi_sw128() { return (1024u >> 4) | (1u << 14) | (2u << 29); }
// MN-major operand in 64-byte rows of 32 elements, one row per k, entries
// permuted (entry ^ (row / 2) % 4); groups of 8 rows are 512 bytes apart, the
// leading offset is the step to the next 32 elements; a K step of 16 is 1024
// bytes.
__device__ __forceinline__ uint32_t umma_hi_mn_sw64() { return (512u >> 4) | (1u << 14) | (4u << 29); }
__device__ __forceinline__ void mma_bf16_lead(uint32_t tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                              uint32_t idesc, uint32_t acc, uint32_t lead) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\t"
        "setp.ne.b32 p, %6, 0;\n\tsetp.ne.b32 q, %7, 0;\n\t"
        "mov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %4};\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}"
        :
        : "r"(tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(acc), "r"(lead)
        : "memory");
}
__device__ __forceinline__ void mma_commit_lead(uint64_t* bar, uint32_t lead) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar)),
        "r"(lead)
        : "memory");
}

// arrive on bar once every MMA issued so far by this thread has completed
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t addr, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(addr), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ bool mbar_wait_bounded(uint32_t addr, uint32_t parity) {
    if (mbar_try(addr, parity)) return true;
    const long long t0 = clock64();
    while (!mbar_try(addr, parity)) {
        if (clock64() - t0 > WAIT_CYCLES) return false;
    }
    return true;
}

__device__ __forceinline__ void cp_async16(uint32_t saddr, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(saddr), "l"(src), "r"(src_bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// bar gets one arrival of this thread once all its cp.async copies so far have
// landed.  The thread itself does not wait, and needs no proxy fence: the
// reader fences after its wait (a fence here would first wait for every copy
// the thread has in flight, i.e. undo the ring).
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// after a wait for copied data: order it before this thread's MMAs
__device__ __forceinline__ void fence_copied() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// 32 TMEM columns of the calling warp's 32 lanes, without the wait
__device__ __forceinline__ void tmem_load32(uint32_t addr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(addr));
}
// COLS (a multiple of 32) accumulator columns as floats, complete on return
template <int COLS> __device__ __forceinline__ void tmem_load(uint32_t addr, float (&v)[COLS]) {
    uint32_t r[COLS / 32][32];
#pragma unroll
    for (int k = 0; k < COLS / 32; k++) tmem_load32(addr + uint32_t(32 * k), r[k]);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < COLS; k++) v[k] = __uint_as_float(r[k / 32][k % 32]);
}

}  // namespace glide
