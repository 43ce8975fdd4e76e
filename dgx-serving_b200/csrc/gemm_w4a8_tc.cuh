// W4A8 prefill GEMM for sm_100a on the 5th-generation tensor cores: the N-sharded GEMM with peer stores and the group-dot dump.
// (On one GPU gemm_w4a8_mma.cuh is faster for every shape.)
//   Y[m,n] = sum_b ((float)D[m,n,b] * xs[m,b]) * sw[n,b],   D[m,n,b] = sum_{k in group b} X[m,k]*(Wq[n,k]-8)
// Semantics and fp32 evaluation order of the reference's kernels/gemm_mmq.cuh:38-120 (t = (float)c*xs,
// acc = fma(t, sw, acc), groups ascending, :104-105), shared by gemm_mma.cuh, gemm_mmq_tmpl.cuh,
// gemm_mmq_raster.cuh and gemm_mmq_ms.cuh.  Because both operands carry a scale per 32-element group,
// the tensor core can only produce ONE group's int32 dot per MMA (K = 32); the scaling and the sum over
// groups run on the CUDA cores, and that epilogue — three lane-operations per (m,n,group) — bounds the
// kernel, not the MMA rate.
//
// Persistent kernel, one CTA per SM, 128x128 output tile per step, warp-specialised:
//   warp 0      TMA producer: int8 activations [128 x 128 B] (128-byte swizzle) and packed int4 weights
//               [128 x 64 B] per K-tile of 128 elements, each behind its own mbarrier ring
//   warp 1      MMA issuer: one tcgen05.mma kind::i8 (128x128x32) per group into one of four 128-column
//               accumulator buffers in tensor memory; tcgen05.commit signals operand release / result ready
//   warps 2-3   expand int4 -> int8 (as 16*(w-8), see unpack8_x16) from the packed stage into the swizzled
//               K-major operand stage the MMA reads (generic-proxy writes + fence.proxy.async), and stage
//               both scale slices of the K-tile in shared memory: weight scales transposed to [group][n] and
//               pre-multiplied by the exact 1/16, activation scales transposed to [group][m]
//   warps 4-19  epilogue: tcgen05.ld the int32 group dots (lane = row, 32 columns per warp, loaded as two
//               16-column chunks so that one chunk's load is in flight while the other is processed), convert,
//               scale and accumulate in registers; store the fp32 tile at the end of the K loop.  The loop
//               touches no global memory.  Sixteen warps rather than eight because each warp's instruction
//               stream is a chain of waits (tensor-memory load, barrier, conversion pipe): four epilogue
//               warps per scheduler overlap them better than two (1253 -> 1214 us at M = 2048).
// Ragged M, N and a last partial K-tile are handled by TMA zero fill plus guards on scales and stores.
#pragma once
#include <cuda.h>
#include "common.cuh"
#include "ptx_sm100.cuh"
#include "peer_allgather.cuh"
#include "tmap_cache.cuh"

namespace w4a8 {
namespace gemm {

constexpr int BM = 128, BN = 128, KT = 128;
constexpr int GPK = KT / QBLK;  // groups (MMAs) per K-tile = 4
#ifndef W4A8_GEMM_SA
#define W4A8_GEMM_SA 4
#endif
#ifndef W4A8_GEMM_SB
#define W4A8_GEMM_SB 4
#endif
constexpr int SA = W4A8_GEMM_SA;  // activation stages
constexpr int SB = W4A8_GEMM_SB;  // packed-weight stages
constexpr int S8 = 3;           // expanded-weight stages
constexpr int SS = 4;           // weight-scale stages
constexpr int TB = 4;           // TMEM accumulator buffers (TB * BN = 512 columns = all of tensor memory)
constexpr int A_STAGE = BM * KT;       // 16 KB
constexpr int BP_STAGE = BN * KT / 2;  // 8 KB
constexpr int B8_STAGE = BN * KT;      // 16 KB
constexpr int SW_STAGE = GPK * (BN + BM) * 4; // 4 KB: weight scales [group][n], then activation scales [group][m]
#ifndef W4A8_DEQ_WARPS
#define W4A8_DEQ_WARPS 2
#endif
#ifndef W4A8_EPI_UNROLL
#define W4A8_EPI_UNROLL 4
#endif
#ifndef W4A8_EPI_WARPS
#define W4A8_EPI_WARPS 16
#endif
constexpr int DEQ_WARPS = W4A8_DEQ_WARPS, EPI_WARPS = W4A8_EPI_WARPS;
constexpr int EPI_UNROLL = W4A8_EPI_UNROLL;
constexpr int EPI_COLS = BN / (EPI_WARPS / 4);  // accumulator columns per epilogue warp (32)
constexpr int EPI_CH = EPI_COLS / 2;           // columns per tcgen05.ld chunk (16)
constexpr int THREADS = (2 + DEQ_WARPS + EPI_WARPS) * 32;  // 640: up to 96 registers per thread
constexpr int OFF_A = 0;
constexpr int OFF_B8 = OFF_A + SA * A_STAGE;
constexpr int OFF_BP = OFF_B8 + S8 * B8_STAGE;
constexpr int OFF_SW = OFF_BP + SB * BP_STAGE;
constexpr int OFF_BAR = OFF_SW + SS * SW_STAGE;
constexpr int NUM_BARS = 2 * (SA + SB + S8 + SS + TB);
constexpr int OFF_TMEM = OFF_BAR + NUM_BARS * 8;
constexpr int SMEM_BYTES = OFF_TMEM + 16 + 1024;  // + slack to align the base to 1024 B

// Device error codes (w4a8_device_status detail): 0x100 | role << 4 | which wait.
enum : unsigned { ERR_PRODUCER = 0x110, ERR_MMA = 0x120, ERR_DEQUANT = 0x130, ERR_EPILOGUE = 0x140 };

struct Ring {
    int stage = 0;
    uint32_t phase = 0;
    const int depth;
    __device__ explicit Ring(int d) : depth(d) {}
    __device__ __forceinline__ void advance() {
        if (++stage == depth) { stage = 0; phase ^= 1u; }
    }
};

// ---- epilogue arithmetic on one chunk of NC accumulator columns ------------------------------------
// d[j] = 16 * D[m, n_j, b] (int32 from tensor memory), x = xs[m,b], sw16[j] = sw[n_j,b] / 16.
// Evaluates t = (float)d * x (rounded), acc = fma(t, sw16, acc): bit-identical to the reference's
// (float)c * xs * sw accumulation (kernels/gemm_mmq.cuh:104-105) because the two factors of 16 are exact.
//   EPI bit 0: int -> float by adding the integer to the bit pattern of 1.5 * 2^23 and subtracting that
//              constant as a float (exact for |d| < 2^22; here |d| <= 520,192) instead of cvt.rn.f32.s32
//   EPI bit 1: packed two-wide fp32 multiply / fma (mul.rn.f32x2, fma.rn.f32x2): same IEEE results per lane
__device__ __forceinline__ float cvt_exact(uint32_t d, bool magic) {
    if (magic) return __int_as_float((int)d + 0x4B400000) - 12582912.0f;
    return __int2float_rn((int)d);
}
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
template <int EPI, int NC>
__device__ __forceinline__ void epi_chunk(const uint32_t (&d)[NC], float x, const float *__restrict__ sw16, float *__restrict__ acc) {
    constexpr bool PACKED = (EPI & 2) != 0, MIXED = (EPI & 4) != 0;
    if (PACKED) {
        const uint64_t xx = pack_f32x2(x, x);
#pragma unroll
        for (int j4 = 0; j4 < NC / 4; j4++) {
            const float4 s4 = *reinterpret_cast<const float4 *>(sw16 + j4 * 4);
            // EPI bit 2: alternate between the two conversions so that neither the conversion pipe nor the
            // fp32 pipe carries all of them
            const bool MAGIC = MIXED ? ((j4 & 1) != 0) : ((EPI & 1) != 0);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int j = j4 * 4 + 2 * h;
                uint64_t f2;
                if (MAGIC) {
                    const uint64_t i2 = pack_f32x2(__int_as_float((int)d[j] + 0x4B400000), __int_as_float((int)d[j + 1] + 0x4B400000));
                    const uint64_t c2 = pack_f32x2(-12582912.0f, -12582912.0f);
                    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(f2) : "l"(i2), "l"(c2));
                } else {
                    f2 = pack_f32x2(__int2float_rn((int)d[j]), __int2float_rn((int)d[j + 1]));
                }
                const uint64_t s2 = h == 0 ? pack_f32x2(s4.x, s4.y) : pack_f32x2(s4.z, s4.w);
                uint64_t a2 = pack_f32x2(acc[j], acc[j + 1]);
                uint64_t t2;
                asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(t2) : "l"(f2), "l"(xx));
                asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(a2) : "l"(t2), "l"(s2));
                unpack_f32x2(a2, acc[j], acc[j + 1]);
            }
        }
    } else {
        constexpr bool MAGIC = (EPI & 1) != 0;
#pragma unroll
        for (int j4 = 0; j4 < NC / 4; j4++) {
            const float4 s4 = *reinterpret_cast<const float4 *>(sw16 + j4 * 4);
            const int j = j4 * 4;
            const float t0 = cvt_exact(d[j + 0], MAGIC) * x;
            const float t1 = cvt_exact(d[j + 1], MAGIC) * x;
            const float t2 = cvt_exact(d[j + 2], MAGIC) * x;
            const float t3 = cvt_exact(d[j + 3], MAGIC) * x;
            acc[j + 0] = fmaf(t0, s4.x, acc[j + 0]);
            acc[j + 1] = fmaf(t1, s4.y, acc[j + 1]);
            acc[j + 2] = fmaf(t2, s4.z, acc[j + 2]);
            acc[j + 3] = fmaf(t3, s4.w, acc[j + 3]);
        }
    }
}
// Four consecutive scales of one row (one K-tile's worth) with one load; the address must be aligned to the
// size of the load.
__device__ __forceinline__ void load_scales4(const float *p, float (&v)[4]) {
    const float4 t = __ldg(reinterpret_cast<const float4 *>(p));
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
__device__ __forceinline__ void load_scales4(const __half *p, float (&v)[4]) {
    const uint2 t = __ldg(reinterpret_cast<const uint2 *>(p));
    const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&t.x));
    const float2 b = __half22float2(*reinterpret_cast<const __half2 *>(&t.y));
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
// Debug path: the exact group dots of one chunk to Dout[m][n][b] (undoing the factor 16).
template <int NC>
__device__ __forceinline__ void epi_dump(const uint32_t (&d)[NC], int32_t *__restrict__ Dout, int m, int M, int ncol0, int N,
                                         int nb, int b) {
    if (m >= M) return;
#pragma unroll
    for (int j = 0; j < NC; j++) {
        const int n = ncol0 + j;
        if (n < N) Dout[((size_t)m * N + n) * nb + b] = ((int)d[j]) >> 4;
    }
}

// One unit of work = (output tile, K split).  Tiles are numbered M-fastest so that CTAs running at the
// same time share weight tiles in L2; split s covers groups [s*gsplit, min(nb, (s+1)*gsplit)).
// Rows [m0, mend) of the tile are live.
struct Work {
    int m0, mend, n0, g0, g1, nkt, split;
};
__device__ __forceinline__ Work decode_work(int w, int m_tiles, int num_tiles, int nb, int gsplit, int M) {
    Work k;
    const int tile = w % num_tiles;
    k.split = w / num_tiles;
    k.m0 = (tile % m_tiles) * BM;
    k.mend = M;
    k.n0 = (tile / m_tiles) * BN;
    k.g0 = k.split * gsplit;
    k.g1 = min(nb, k.g0 + gsplit);
    const int ng = max(0, k.g1 - k.g0);
    k.nkt = (ng + GPK - 1) / GPK;
    return k;
}

// PEER (N-sharded weights, no split-K): every output tile is stored straight into EVERY rank's Y[M, ld] at its final
// columns (oa.col0 + n: plain 16-byte peer stores over NVLink) and the last CTA publishes the step's epoch, so the
// all-gather costs no extra pass over the outputs (peer_allgather.cuh).
template <typename ST, bool DUMP, int EPI, bool PEER = false>
__global__ void __launch_bounds__(THREADS, 1) gemm_w4a8_tc_kernel(
    const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
    const float *__restrict__ xs, const ST *__restrict__ sw, float *__restrict__ Y, int32_t *__restrict__ Dout,
    int M, int N, int K, int nsplit, int gsplit, const OutArgs oa) {
    extern __shared__ unsigned char smem_dyn[];
    const uint32_t raw = ptx::smem_u32(smem_dyn);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char *base_ptr = smem_dyn + (base - raw);

    const uint32_t bar0 = base + OFF_BAR;
    auto BAR = [&](int idx) { return bar0 + 8u * idx; };
    // barrier index map
    constexpr int A_FULL = 0, A_EMPTY = A_FULL + SA, BP_FULL = A_EMPTY + SA, BP_EMPTY = BP_FULL + SB,
                  B8_FULL = BP_EMPTY + SB, B8_EMPTY = B8_FULL + S8, SW_FULL = B8_EMPTY + S8, SW_EMPTY = SW_FULL + SS,
                  TM_FULL = SW_EMPTY + SS, TM_EMPTY = TM_FULL + TB;
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(base_ptr + OFF_TMEM);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nb = K / QBLK;
    const bool scales_aligned = ((reinterpret_cast<uintptr_t>(xs) & 15) == 0) && ((reinterpret_cast<uintptr_t>(sw) & (4 * sizeof(ST) - 1)) == 0);
    const int m_tiles = (M + BM - 1) / BM, n_tiles = (N + BN - 1) / BN;
    const int num_tiles = m_tiles * n_tiles;
    const int num_work = num_tiles * nsplit;

    if (tid == 0) {
        for (int i = 0; i < SA; i++) { ptx::mbar_init(BAR(A_FULL + i), 1); ptx::mbar_init(BAR(A_EMPTY + i), 1); }
        for (int i = 0; i < SB; i++) { ptx::mbar_init(BAR(BP_FULL + i), 1); ptx::mbar_init(BAR(BP_EMPTY + i), DEQ_WARPS); }
        for (int i = 0; i < S8; i++) { ptx::mbar_init(BAR(B8_FULL + i), DEQ_WARPS); ptx::mbar_init(BAR(B8_EMPTY + i), 1); }
        for (int i = 0; i < SS; i++) { ptx::mbar_init(BAR(SW_FULL + i), DEQ_WARPS); ptx::mbar_init(BAR(SW_EMPTY + i), EPI_WARPS); }
        for (int i = 0; i < TB; i++) { ptx::mbar_init(BAR(TM_FULL + i), 1); ptx::mbar_init(BAR(TM_EMPTY + i), EPI_WARPS); }
        ptx::mbar_fence_init();
        ptx::tma_prefetch_desc(&tmA);
        ptx::tma_prefetch_desc(&tmB);
    }
    if (warp == 1) {
        ptx::tmem_alloc(ptx::smem_u32(const_cast<uint32_t *>(tmem_slot)), TB * BN);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before_sync();
    __syncthreads();
    ptx::tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            Ring ra(SA), rb(SB);
            bool ok = true;
            for (int wi = blockIdx.x; wi < num_work && ok; wi += gridDim.x) {
                const Work wk = decode_work(wi, m_tiles, num_tiles, nb, gsplit, M);
                const int m0 = wk.m0, n0 = wk.n0;
                for (int kt = 0; kt < wk.nkt && ok; kt++) {
                    const int kbyte = (wk.g0 + kt * GPK) * QBLK;   // first K element of this K-tile (multiple of 32)
                    if (!ptx::mbar_wait(BAR(A_EMPTY + ra.stage), ra.phase ^ 1u)) { dev_set_error(ERR_PRODUCER | 1); ok = false; break; }
                    ptx::mbar_arrive_expect_tx(BAR(A_FULL + ra.stage), A_STAGE);
                    ptx::tma_load_2d(base + OFF_A + ra.stage * A_STAGE, &tmA, kbyte, m0, BAR(A_FULL + ra.stage));
                    ra.advance();
                    if (!ptx::mbar_wait(BAR(BP_EMPTY + rb.stage), rb.phase ^ 1u)) { dev_set_error(ERR_PRODUCER | 2); ok = false; break; }
                    ptx::mbar_arrive_expect_tx(BAR(BP_FULL + rb.stage), BP_STAGE);
                    ptx::tma_load_2d(base + OFF_BP + rb.stage * BP_STAGE, &tmB, kbyte / 2, n0, BAR(BP_FULL + rb.stage));
                    rb.advance();
                }
            }
            if (!ok) {  // give copies already in flight time to land before the CTA's shared memory goes away
                const long long t0 = clock64();
                while (clock64() - t0 < (1ll << 21)) { }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        if (lane == 0) {
            Ring ra(SA), r8(S8), rt(TB);
            const uint32_t idesc = ptx::umma_idesc_s8(BM, BN);
            bool ok = true;
            for (int wi = blockIdx.x; wi < num_work && ok; wi += gridDim.x) {
                const Work wk = decode_work(wi, m_tiles, num_tiles, nb, gsplit, M);
                for (int kt = 0; kt < wk.nkt && ok; kt++) {
                    if (!ptx::mbar_wait(BAR(A_FULL + ra.stage), ra.phase)) { dev_set_error(ERR_MMA | 1); ok = false; break; }
                    if (!ptx::mbar_wait(BAR(B8_FULL + r8.stage), r8.phase)) { dev_set_error(ERR_MMA | 2); ok = false; break; }
                    ptx::tc_fence_after_sync();
                    const uint64_t adesc = ptx::umma_desc_k_sw128(base + OFF_A + ra.stage * A_STAGE);
                    const uint64_t bdesc = ptx::umma_desc_k_sw128(base + OFF_B8 + r8.stage * B8_STAGE);
                    const int ng = min(GPK, wk.g1 - (wk.g0 + kt * GPK));
                    for (int g = 0; g < ng; g++) {
                        if (!ptx::mbar_wait(BAR(TM_EMPTY + rt.stage), rt.phase ^ 1u)) { dev_set_error(ERR_MMA | 3); ok = false; break; }
                        ptx::tc_fence_after_sync();
                        // group g = bytes [32g, 32g+32) of every 128-byte operand row: advance the start address
                        ptx::umma_i8(tmem_base + rt.stage * BN, adesc + (uint64_t)(g * 2), bdesc + (uint64_t)(g * 2), idesc, 0u);
                        ptx::umma_commit(BAR(TM_FULL + rt.stage));
                        rt.advance();
                    }
                    ptx::umma_commit(BAR(A_EMPTY + ra.stage));
                    ptx::umma_commit(BAR(B8_EMPTY + r8.stage));
                    ra.advance();
                    r8.advance();
                }
            }
        }
    } else if (warp < 2 + DEQ_WARPS) {
        // ---------------- int4 -> int8 expansion + weight-scale staging ----------------
        const int dt = tid - 64;  // 0..DEQ_WARPS*32-1
        Ring rb(SB), r8(S8), rs(SS);
        bool ok = true;
        for (int wi = blockIdx.x; wi < num_work && ok; wi += gridDim.x) {
            const Work wk = decode_work(wi, m_tiles, num_tiles, nb, gsplit, M);
            const int n0 = wk.n0;
            for (int kt = 0; kt < wk.nkt && ok; kt++) {
                // ---- this K-tile's scales: issue the loads first, they complete behind the expansion below.
                // A row's GPK scales are contiguous in memory: one 16-byte (fp32) or 8-byte (fp16) load per row
                // when the K-tile is complete and the addresses line up, else element by element.
                constexpr int RW = BN / (DEQ_WARPS * 32), RX = BM / (DEQ_WARPS * 32);
                const int b0 = wk.g0 + kt * GPK;   // first group of this K-tile
                const bool vec = !DUMP && (b0 + GPK <= wk.g1) && (nb % GPK == 0) && (b0 % GPK == 0) && scales_aligned;
                float vw[RW][GPK], vx[RX][GPK];
#pragma unroll
                for (int r = 0; r < RW; r++) {
                    const int n = n0 + dt + r * DEQ_WARPS * 32;
#pragma unroll
                    for (int g = 0; g < GPK; g++) vw[r][g] = 0.f;
                    if (!DUMP && n < N) {
                        const ST *swrow = sw + (size_t)n * nb;
                        if (vec) load_scales4(swrow + b0, vw[r]);
                        else {
#pragma unroll
                            for (int g = 0; g < GPK; g++)
                                if (b0 + g < wk.g1) vw[r][g] = sval(swrow[b0 + g]);
                        }
                    }
                }
#pragma unroll
                for (int r = 0; r < RX; r++) {
                    const int m = wk.m0 + dt + r * DEQ_WARPS * 32;
#pragma unroll
                    for (int g = 0; g < GPK; g++) vx[r][g] = 0.f;
                    if (!DUMP && m < wk.mend) {
                        if (vec) load_scales4(xs + (size_t)m * nb + b0, vx[r]);
                        else {
#pragma unroll
                            for (int g = 0; g < GPK; g++)
                                if (b0 + g < wk.g1) vx[r][g] = xs[(size_t)m * nb + b0 + g];
                        }
                    }
                }

                // ---- expansion of the packed stage into the operand stage
                bool w = ptx::mbar_wait_warp(BAR(BP_FULL + rb.stage), rb.phase) && ptx::mbar_wait_warp(BAR(B8_EMPTY + r8.stage), r8.phase ^ 1u);
                if (!w) { dev_set_error(ERR_DEQUANT | 1); ok = false; break; }
                const unsigned char *src = base_ptr + OFF_BP + rb.stage * BP_STAGE;
                unsigned char *dst = base_ptr + OFF_B8 + r8.stage * B8_STAGE;
                // All loads first, then expansion and stores: the compiler cannot tell that the two stages do not
                // overlap, so in one loop every load would wait for the previous store.
                constexpr int NT = (BN * 8) / (DEQ_WARPS * 32);
                uint2 pk[NT];
#pragma unroll
                for (int i = 0; i < NT; i++) {
                    const int j = dt + i * DEQ_WARPS * 32;
                    const int n = j >> 3, c = j & 7;  // row n, 8 packed bytes = 16 weights = one 16-byte chunk
                    pk[i] = *reinterpret_cast<const uint2 *>(src + n * (KT / 2) + c * 8);
                }
#pragma unroll
                for (int i = 0; i < NT; i++) {
                    const int j = dt + i * DEQ_WARPS * 32;
                    const int n = j >> 3, c = j & 7;
                    uint4 o;
                    unpack8_x16_seq(pk[i].x, o.x, o.y);
                    unpack8_x16_seq(pk[i].y, o.z, o.w);
                    *reinterpret_cast<uint4 *>(dst + n * KT + ((c ^ (n & 7)) << 4)) = o;
                }
                ptx::fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) { ptx::mbar_arrive(BAR(B8_FULL + r8.stage)); ptx::mbar_arrive(BAR(BP_EMPTY + rb.stage)); }
                rb.advance();
                r8.advance();

                // ---- store the scales: weight scales transposed to [group][n] and pre-multiplied by the exact
                // 1/16 that undoes the 16x of the expansion, activation scales transposed to [group][m]
                w = ptx::mbar_wait_warp(BAR(SW_EMPTY + rs.stage), rs.phase ^ 1u);
                if (!w) { dev_set_error(ERR_DEQUANT | 2); ok = false; break; }
                float *ssw = reinterpret_cast<float *>(base_ptr + OFF_SW + rs.stage * SW_STAGE);
                float *ssx = ssw + GPK * BN;
#pragma unroll
                for (int r = 0; r < RW; r++)
#pragma unroll
                    for (int g = 0; g < GPK; g++) ssw[g * BN + dt + r * DEQ_WARPS * 32] = vw[r][g] * 0.0625f;
#pragma unroll
                for (int r = 0; r < RX; r++)
#pragma unroll
                    for (int g = 0; g < GPK; g++) ssx[g * BM + dt + r * DEQ_WARPS * 32] = vx[r][g];
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(BAR(SW_FULL + rs.stage));
                rs.advance();
            }
        }
    } else {
        // ---------------- epilogue ----------------
        const int ew = warp - (2 + DEQ_WARPS);  // 0..EPI_WARPS-1
        const int quad = warp & 3;              // TMEM lanes [32*quad, 32*quad+32) are the ones this warp may read
        const int col0 = (ew >> 2) * EPI_COLS;  // this warp's accumulator columns [col0, col0 + EPI_COLS)
        Ring rs(SS), rt(TB);
        bool ok = true;
        for (int wi = blockIdx.x; wi < num_work && ok; wi += gridDim.x) {
            const Work wk = decode_work(wi, m_tiles, num_tiles, nb, gsplit, M);
            const int m0 = wk.m0, n0 = wk.n0;
            const int m = m0 + quad * 32 + lane;
            // a warp whose 32 rows all lie beyond M only keeps the barriers moving
            const bool rows_live = (m0 + quad * 32) < wk.mend;
            float acc[EPI_COLS];
#pragma unroll
            for (int j = 0; j < EPI_COLS; j++) acc[j] = 0.f;
            const int ngroups = wk.g1 - wk.g0;
            const uint32_t tlane = tmem_base + ((uint32_t)(quad * 32) << 16) + col0;
            // One flat loop over the groups of this unit of work.  The 2 chunks (EPI_CH columns each) of a group
            // are software-pipelined with the next group's: the tcgen05.ld of the next chunk is in flight while
            // the current one is converted and accumulated.  d0 holds the first half of this warp's columns of
            // a group, d1 the second.  Both scales come from the staged K-tile slice in shared memory, so the
            // loop issues no global loads.
            uint32_t d0[EPI_CH], d1[EPI_CH];
            const float *ssw = nullptr, *ssx = nullptr;
            bool w = true;
            if (ngroups > 0) {   // a split beyond the last group has no work: its partial sums are zeros
                w = ptx::mbar_wait_warp(BAR(TM_FULL + rt.stage), rt.phase);
                if (!w) { dev_set_error(ERR_EPILOGUE | 2); ok = false; break; }
                ptx::tc_fence_after_sync();
                if (rows_live) ptx::tmem_ld(tlane + rt.stage * BN, d0);
            }
#pragma unroll EPI_UNROLL
            for (int gi = 0; gi < ngroups; gi++) {
                const int g = gi & (GPK - 1);
                if (g == 0) {
                    w = ptx::mbar_wait_warp(BAR(SW_FULL + rs.stage), rs.phase);
                    if (!w) { dev_set_error(ERR_EPILOGUE | 1); ok = false; break; }
                    ssw = reinterpret_cast<const float *>(base_ptr + OFF_SW + rs.stage * SW_STAGE) + col0;
                    ssx = reinterpret_cast<const float *>(base_ptr + OFF_SW + rs.stage * SW_STAGE) + GPK * BN + quad * 32 + lane;
                }
                const float x = ssx[g * BM];
                const uint32_t tcur = tlane + rt.stage * BN;
                // ---- first half: wait for it, start the second half's load, then compute
                ptx::tmem_ld_wait();
                if (rows_live) ptx::tmem_ld(tcur + EPI_CH, d1);
                if (rows_live) {
                    if (DUMP) epi_dump<EPI_CH>(d0, Dout, m, wk.mend, n0 + col0, N, nb, wk.g0 + gi);
                    else epi_chunk<EPI, EPI_CH>(d0, x, ssw + g * BN, acc);
                }
                // ---- second half: wait, release the accumulator buffer, start the next group's load
                ptx::tmem_ld_wait();
                ptx::tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(BAR(TM_EMPTY + rt.stage));
                rt.advance();
                if (gi + 1 < ngroups) {
                    w = ptx::mbar_wait_warp(BAR(TM_FULL + rt.stage), rt.phase);
                    if (!w) { dev_set_error(ERR_EPILOGUE | 3); ok = false; break; }
                    ptx::tc_fence_after_sync();
                    if (rows_live) ptx::tmem_ld(tlane + rt.stage * BN, d0);
                }
                if (rows_live) {
                    if (DUMP) epi_dump<EPI_CH>(d1, Dout, m, wk.mend, n0 + col0 + EPI_CH, N, nb, wk.g0 + gi);
                    else epi_chunk<EPI, EPI_CH>(d1, x, ssw + g * BN + EPI_CH, acc + EPI_CH);
                }
                if (g == GPK - 1 || gi + 1 == ngroups) {   // done with this K-tile's scales
                    __syncwarp();
                    if (lane == 0) ptx::mbar_arrive(BAR(SW_EMPTY + rs.stage));
                    rs.advance();
                }
            }
            if (!ok) break;
            if (!DUMP && ok && m < wk.mend) {
                const int nleft = N - (n0 + col0);
                const int targets = PEER ? oa.peers->world : 1;
                for (int k = 0; k < targets; k++) {
                    if (PEER && oa.local_only && k != oa.peers->rank) continue;
                    float *yrow = PEER ? reinterpret_cast<float *>(oa.peers->base[k] + oa.y_off) + (size_t)m * oa.ld + oa.col0 + n0 + col0
                                       : Y + (size_t)wk.split * ((size_t)M * N) + (size_t)m * N + n0 + col0;
                    if (nleft >= EPI_COLS && ((reinterpret_cast<uintptr_t>(yrow) & 15) == 0)) {
#pragma unroll
                        for (int j = 0; j < EPI_COLS; j += 4)
                            *reinterpret_cast<float4 *>(yrow + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
                    } else {
#pragma unroll
                        for (int j = 0; j < EPI_COLS; j++)
                            if (j < nleft) yrow[j] = acc[j];
                    }
                }
            }
        }
    }

    publish_out<PEER>(oa, warp >= 2 + DEQ_WARPS);
    // ---------------- teardown ----------------
    ptx::tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        ptx::tc_fence_after_sync();
        ptx::tmem_dealloc(tmem_base, TB * BN);
    }
}

// Adds the split-K partial sums in ascending split order (the order of the reference's
// reduce_splitk_kernel, kernels/gemm_mmq.cuh:201-204): Y[i] = ((0 + P0[i]) + P1[i]) + ...
// VEC: float or float4 (MN a multiple of four, both pointers aligned).  Launched dependent: it waits at once, but its launch latency
// hides behind the end of the product.
template <typename VEC>
__global__ void __launch_bounds__(256) splitk_reduce_kernel(const VEC *__restrict__ P, VEC *__restrict__ Y, long n, int nsplit) {
    const long stride = (long)gridDim.x * blockDim.x;
    pdl_wait();
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        if constexpr (sizeof(VEC) == 16) {
            float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
            for (int sp = 0; sp < nsplit; sp++) {
                const float4 v = P[(size_t)sp * n + i];
                s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
            }
            Y[i] = s;
        } else {
            float s = 0.f;                               // unrolled by the compiler: by a pragma 21 x 584 x 512 in eight ranges 3.8 us, 3.5 so
            for (int sp = 0; sp < nsplit; sp++) s += P[(size_t)sp * n + i];
            Y[i] = s;
        }
    }
}
inline int launch_splitk_reduce(const float *P, float *Y, long MN, int nsplit, cudaStream_t st) {
    // Four columns a thread where single ones would be more than four CTAs per SM.  us of the whole product, one / four: 21 x 584 x 512 in
    // eight ranges 3.5 / 4.0, 52 x 162 x 2560 4.8 / 5.3, 16 x 5120 x 5120 in eight 9.2 / 9.5, 100 x 1024 x 4096 in four 8.7 / 8.6,
    // 64 x 3840 x 3840 in four 12.6 / 12.2, 300 x 2000 x 4096 in two 25.3 / 24.4.
    const bool vec = MN > 4L * 256 * sm_count() && MN % 4 == 0 && aligned(P, 16) && aligned(Y, 16);
    const long n = vec ? MN / 4 : MN, want = (n + 255) / 256, cap = (long)sm_count() * 8;
    const dim3 grid((unsigned)(want < cap ? want : cap));
    const cudaError_t e = vec ? launch_pdl(splitk_reduce_kernel<float4>, grid, dim3(256), 0, st, reinterpret_cast<const float4 *>(P), reinterpret_cast<float4 *>(Y), n, nsplit)
                              : launch_pdl(splitk_reduce_kernel<float>, grid, dim3(256), 0, st, P, Y, n, nsplit);
    if (e != cudaSuccess) return cuda_fail(e, "splitk_reduce launch");
    return launch_status("splitk_reduce");
}

// ---- host side ------------------------------------------------------------------------------------
template <typename ST, bool DUMP, int EPI, bool PEER = false>
inline int launch_tc_e(const int8_t *X, const float *xs, const uint8_t *Wq, const ST *sw, float *Y, int32_t *D,
                       int M, int N, int K, int nsplit, int gsplit, cudaStream_t st, const OutArgs &oa) {
    CUtensorMap tmA, tmB;
    int rc = make_tmap_u8(&tmA, X, (uint64_t)K, (uint64_t)M, KT, BM, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc != W4A8_OK) return rc;
    rc = make_tmap_u8(&tmB, Wq, (uint64_t)K / 2, (uint64_t)N, KT / 2, BN, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (rc != W4A8_OK) return rc;
    auto kern = gemm_w4a8_tc_kernel<ST, DUMP, EPI, PEER>;
    static PerDevice<bool> configured_dev;              // the opt-in is a per-device function attribute
    bool &configured = configured_dev.get();
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
        if (e != cudaSuccess) return cuda_fail(e, "gemm smem opt-in");
        configured = true;
    }
    const long tiles = (long)((M + BM - 1) / BM) * ((N + BN - 1) / BN) * nsplit;
    const int sms = sm_count();
    const unsigned grid = (unsigned)(tiles < sms ? tiles : sms);
    kern<<<grid, THREADS, SMEM_BYTES, st>>>(tmA, tmB, xs, sw, Y, D, M, N, K, nsplit, gsplit, PEER ? oa : OutArgs());
    return launch_status("gemm_w4a8_tc");
}

// Needs X and Wq 16-byte aligned (TMA global address rule); the caller checks.
// Epilogue arithmetic variant (see epi_chunk): all variants give identical bits.  W4A8_GEMM_EPI overrides the
// default for measurements (0 cvt, 1 magic-number conversion, 2 cvt + f32x2, 3 magic + f32x2).
inline int epi_variant() {
    static int v = -1;
    if (v < 0) {
        const char *e = getenv("W4A8_GEMM_EPI");
        v = e ? atoi(e) & 7 : 2;
    }
    return v;
}
template <typename ST, bool DUMP>
inline int launch_tc_t(const int8_t *X, const float *xs, const uint8_t *Wq, const ST *sw, float *Y, int32_t *D,
                       int M, int N, int K, int nsplit, int gsplit, cudaStream_t st, const OutArgs &oa) {
    if (!DUMP && oa.peers) return launch_tc_e<ST, false, 2, true>(X, xs, Wq, sw, Y, D, M, N, K, nsplit, gsplit, st, oa);
    switch (DUMP ? 0 : epi_variant()) {
        case 1: return launch_tc_e<ST, DUMP, 1>(X, xs, Wq, sw, Y, D, M, N, K, nsplit, gsplit, st, oa);
        case 2: return launch_tc_e<ST, DUMP, 2>(X, xs, Wq, sw, Y, D, M, N, K, nsplit, gsplit, st, oa);
        case 3: return launch_tc_e<ST, DUMP, 3>(X, xs, Wq, sw, Y, D, M, N, K, nsplit, gsplit, st, oa);
        case 6: return launch_tc_e<ST, DUMP, 6>(X, xs, Wq, sw, Y, D, M, N, K, nsplit, gsplit, st, oa);
        default: return launch_tc_e<ST, DUMP, 0>(X, xs, Wq, sw, Y, D, M, N, K, nsplit, gsplit, st, oa);
    }
}

// nsplit = 1: Y is the output.  nsplit > 1: Y is the [nsplit][M][N] partial-sum workspace and gsplit the
// number of groups per split.
inline int launch_tc(const int8_t *X, const float *xs, const uint8_t *Wq, const void *sw, float *Y, int M, int N, int K,
                     int scale_dtype, int nsplit, int gsplit, cudaStream_t st, const OutArgs &oa = OutArgs()) {
    if (scale_dtype == 1)
        return launch_tc_t<__half, false>(X, xs, Wq, (const __half *)sw, Y, nullptr, M, N, K, nsplit, gsplit, st, oa);
    return launch_tc_t<float, false>(X, xs, Wq, (const float *)sw, Y, nullptr, M, N, K, nsplit, gsplit, st, oa);
}
inline int launch_tc_dump(const int8_t *X, const uint8_t *Wq, int32_t *D, int M, int N, int K, cudaStream_t st) {
    return launch_tc_t<float, true>(X, nullptr, Wq, (const float *)nullptr, nullptr, D, M, N, K, 1, K / QBLK, st, OutArgs());
}

}  // namespace gemm
}  // namespace w4a8
