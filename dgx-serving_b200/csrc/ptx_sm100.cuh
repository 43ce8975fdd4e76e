// Inline-PTX wrappers for the sm_100a features the GEMM uses: mbarrier, TMA (cp.async.bulk.tensor),
// tensor memory (tcgen05.alloc/ld) and the 5th-generation tensor-core MMA (tcgen05.mma kind::i8).
// Every wait is bounded: a wait that runs out records an error code and returns false so that the
// caller can leave its loop; nothing in this file can spin forever.
#pragma once
#include <cstdint>

namespace w4a8 {
namespace ptx {

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ---- mbarrier ----------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// One attempt; comes back after a short system-chosen time if the phase has not completed (about 34 cycles
// when it has).
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Polling loop behind the first attempt.  Kept out of line on purpose: inlined, the 64-bit clock read that
// bounds the loop was scheduled ahead of the first attempt and a wait on a barrier that had ALREADY completed
// cost about 180 cycles instead of 34, on every hand-off of the pipeline.  The clock is read once per 64
// attempts so that it does not delay the wake-up either.  Gives up after `limit_cycles` SM clocks.
// (Passing a suspend-time hint of 2 us to try_wait changed no kernel's time: measured and left out.)
__device__ __noinline__ bool mbar_wait_poll(uint32_t bar, uint32_t parity, long long limit_cycles) {
    const long long t0 = clock64();
    for (;;) {
        for (int i = 0; i < 64; i++)
            if (mbar_try_wait(bar, parity)) return true;
        if (clock64() - t0 > limit_cycles) return false;
    }
}
// Bounded wait of one thread: the default limit of 2^28 cycles (about 0.15 s) is far beyond any legitimate
// pipeline wait (microseconds).  Returns false on timeout.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, long long limit_cycles = (1ll << 28)) {
    if (mbar_try_wait(bar, parity)) return true;
    return mbar_wait_poll(bar, parity, limit_cycles);
}

// Warp-wide bounded wait: every lane makes the attempt (uniform control flow, about 47 cycles with the vote
// when the phase has completed; letting one lane wait and broadcasting the outcome by shuffle cost more) and
// the warp leaves together with one agreed result.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, long long limit_cycles = (1ll << 28)) {
    bool ok = mbar_try_wait(bar, parity);
    if (__all_sync(0xffffffffu, ok)) return true;
    if (!ok) ok = mbar_wait_poll(bar, parity, limit_cycles);
    return __all_sync(0xffffffffu, ok);
}

// ---- proxies / fences -------------------------------------------------------------------------
// Makes generic-proxy shared-memory writes visible to the async proxy (TMA, tcgen05.mma operands).
__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ---- TMA: 2-D tiled load global -> shared, completion on an mbarrier (no multicast) -----------
__device__ __forceinline__ void tma_load_2d(uint32_t dst_smem, const void *tmap, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst_smem), "l"(tmap), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const void *tmap) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(tmap) : "memory");
}
// Brings `bytes` (a multiple of 16) of global memory starting at a 16-byte aligned address into L2; nothing waits for it.
__device__ __forceinline__ void prefetch_l2_bulk(const void *gptr, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(gptr), "r"(bytes) : "memory");
}
// While a kernel waits for the one before it, HBM is idle: about 3 us in a chain of decode steps.  One thread of a CTA asks, ahead of
// its wait, for the first `budget` bytes of the CTA's contiguous rows of weights (and their scales) to be brought to L2.  Nothing
// is read into the SM, so this is safe whatever the kernels before write: their stores meet the lines in L2.
__device__ __forceinline__ void prefetch_rows_l2(const uint8_t *w, const void *s, int rows, uint32_t wrow, uint32_t srow, uint32_t budget) {
    const int fit = (int)(budget / (wrow + srow)), n = rows < fit ? rows : fit;
    if (n <= 0) return;
    const auto range = [](const void *p, uint64_t bytes) {                // the 16-byte pieces inside [p, p + bytes)
        const uint64_t a = (reinterpret_cast<uint64_t>(p) + 15) & ~15ull, e = (reinterpret_cast<uint64_t>(p) + bytes) & ~15ull;
        if (e > a) prefetch_l2_bulk(reinterpret_cast<const void *>(a), (uint32_t)(e - a));
    };
    range(w, (uint64_t)n * wrow);
    range(s, (uint64_t)n * srow);
}

// ---- tensor memory ------------------------------------------------------------------------------
// Whole-warp calls (.sync.aligned).  ncols: power of two in [32, 512].
__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// Each lane i of the warp reads 32 consecutive 32-bit columns of TMEM lane (taddr.lane + i).
__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
// 16-column variant (16 registers per lane).
__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
// Narrow variants: 1, 2, 4 and 8 columns per lane.
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[1]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(r[0]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[2]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[32]) { tmem_ld_32x32b_x32(taddr, r); }
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[16]) { tmem_ld_32x32b_x16(taddr, r); }
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// ---- tcgen05.mma, kind::i8 (int8 x int8 -> int32 in TMEM), one CTA -----------------------------
// Shared-memory matrix descriptor for a K-major operand tile stored with the 128-byte swizzle:
// rows of 128 bytes, 16-byte chunk c of row r at chunk position c ^ (r & 7), 8-row groups 1024 bytes
// apart (stride byte offset), tile base 1024-byte aligned.  Field layout: start address >> 4 in bits
// [0,14), leading byte offset >> 4 in [16,30) (unused for swizzled K-major; 1), stride byte offset >> 4 in
// [32,46), descriptor version 1 in [46,48), swizzle mode 2 (= 128 B) in [61,64).
__device__ __forceinline__ uint64_t umma_desc_k_sw128(uint32_t smem_addr) {
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) |
           (2ull << 61);
}
// Instruction descriptor: D = int32 (c_format 2, bits [4,6)); A, B = signed 8-bit (format 1, bits [7,10) and
// [10,13)); both K-major (bits 15, 16 = 0); N >> 3 in [17,23); M >> 4 in [24,29).
__host__ __device__ constexpr uint32_t umma_idesc_s8(int M, int N) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
// Issued by ONE thread.  accumulate = 0 overwrites D, 1 adds to it.
__device__ __forceinline__ void umma_i8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                        uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrives on the mbarrier once every tcgen05 operation issued so far by this thread has completed.
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

}  // namespace ptx
}  // namespace w4a8
