// W4A8 prefill / verify / grouped-expert GEMM whose group dots never leave the register file.
//   Y[m,n] = sum_b ((float)D[m,n,b] * xs[m,b]) * sw[n,b],   D[m,n,b] = sum_{k in group b} X[m,k]*(Wq[n,k]-8)
// Same semantics and fp32 order as gemm_w4a8_tc.cuh (t = (float)D*xs rounded, acc = fma(t, sw, acc), groups ascending:
// the reference's kernels/gemm_mmq.cuh:104-105), hence the same bits.  The dots come out 16 times too large (unpack8_x16);
// the 1/16 goes into the weight scale, as there, where it is exact from 2^-122 up whatever the activation scale is.
//
// What bounds it.  Both operands carry a scale per 32-element group, so whatever computes the dots, every (m, n, group)
// costs a conversion, a multiply and an fma on the CUDA cores.  On tcgen05 the dots come out in tensor memory and every
// group pays, on top of that, a commit, a barrier, tcgen05.ld and a release through four accumulator buffers: about 950 SM
// cycles per 128 x 128 outputs and group, at 6 % tensor-pipe use, and always for 128 rows.  mma.sync m16n8k32 leaves the
// dots in the registers that the epilogue reads: no hand-off, and a tile has as many rows as there are, in steps of 16.
// Alone (a loop without loads) MMA 314, I2F 337 and packed mul + fma 370 cycles per 128 x 128 group, together about 500;
// with the operand and scale traffic the kernel needs about 840 with 128 x 128 tiles.  It issues on 52 % of the cycles with two
// warps per scheduler; the rest are waits on the register file, the pipes, loads from shared memory and MMA results.
// Measured, us: 2048 x 17408 x 5120 1086 (tcgen05 1213), 512 rows 296 (327), 333 x 15360 x 3840 158 (187), 48 x 3840 x 15360 in
// three K ranges, twice, with the quantizer, 106 (174).  Slower in the first versions, in cycles per 128 x 128 group:
// integer-to-float through a preset accumulator (1.5 * 2^23) instead of I2F (1133 against 989), scalar instead of packed fp32
// (1044 against 864), scales through registers (977 against 864; they spill).
//
// Data flow.  cp.async brings K-tiles of 4 groups into a STAGES-deep ring, laid out [group][row][32 B] for the int8
// activations and [group][row][16 B] for the packed weights, so that a warp's fragment reads are contiguous (LDS.64 and
// LDS.32, no conflicts); groups are 32 bytes further apart than they need, which makes the copies' writes conflict-free
// too.  A lane's word of weights expands to its two B registers with three logic operations (unpack8_x16: even and odd
// elements), the matching A registers are two byte permutes of eight activations.  Any order of K inside a group gives
// the same integer.  Scales travel with their K-tile, [row][group], one 16-byte (fp16: 8-byte) piece per row where they line
// up, that is where K / 32 and every range of a split K are multiples of four and the pointers aligned (VEC); 4 bytes at a
// time otherwise, and fp16 scales of an odd K / 32, whose rows start between two words, by plain loads.  Plain loads of all
// scales stall their warp once per K-tile, which cost more than the kernel gains over tcgen05: 700 x 9000 x 5024 321 us with
// them, 246 on tcgen05.  One __syncthreads per K-tile; two or three CTAs per SM cover each other's.
#pragma once
#include <type_traits>
#include "common.cuh"
#include "gemm_w4a8_tc.cuh"

namespace w4a8 {
namespace gemm_mma {

constexpr int GPK = 4;                    // groups per K-tile
// live = false writes zeros and reads nothing
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// D(16x8, s32) = A(16x32, s8, row) * B(32x8, s8, col)
__device__ __forceinline__ void mma_s8(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ void fma2(uint64_t &acc, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// TM m16 tiles x TN n8 tiles per warp, WM x WN warps, CTAs per SM the register and shared-memory budget is cut for.
template <int TM_, int TN_, int WM_, int WN_, int STAGES_, int CTAS_>
struct Cfg {
    static constexpr int TM = TM_, TN = TN_, WM = WM_, WN = WN_, STAGES = STAGES_, CTAS = CTAS_;
    static constexpr int BM = 16 * TM * WM, BN = 8 * TN * WN, THREADS = 32 * WM * WN;
    static constexpr int A_GROUP = BM * 32 + 32, B_GROUP = BN * 16 + 32;      // bytes; + 32 keeps the copies' writes conflict-free
    static constexpr int OFF_SX = GPK * (A_GROUP + B_GROUP), OFF_SW = OFF_SX + BM * GPK * 4;      // scales: [row][group]
    static constexpr int STAGE = OFF_SW + BN * GPK * 4, SMEM = STAGES * STAGE;
    static constexpr int RB = (BN + THREADS - 1) / THREADS, RA = (BM + THREADS - 1) / THREADS;   // scale rows per thread
    static_assert(CTAS * (SMEM + 1024) <= 228 * 1024, "CTAS of these do not fit an SM's shared memory (1 KB each is the system's)");
};

// Grouped experts: the activation rows are sorted by expert, item i of the list says "expert x, sorted rows [y, y + z)" with
// z <= ITEM_ROWS (one item per 64-row tile of an expert, written on the device by moe_sort_kernel), the weights are the
// flat [experts * N][K/2] tensor of the reference (kernels/moe_fused.cuh:21-24: expert e starts e * N rows in), and one
// unit of work is (item, 128 of the expert's N outputs).
constexpr int ITEM_ROWS = 64;
struct GroupList {
    const int4 *items = nullptr;
    const int *num_items = nullptr;
};

template <class C, typename ST, bool GROUPED, bool VEC>
__global__ void __launch_bounds__(C::THREADS, C::CTAS) gemm_w4a8_mma_kernel(
    const int8_t *__restrict__ X, const float *__restrict__ xs, const uint8_t *__restrict__ Wq, const ST *__restrict__ sw,
    float *__restrict__ Y, int M, int N, int K, int m_tiles, int n_tiles, int gsplit, bool pairs, const GroupList gl) {
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr int TM = C::TM, TN = C::TN, BM = C::BM, BN = C::BN, NT = C::THREADS, STAGES = C::STAGES;
    // Scales that line up make every K-tile complete.  Known at compile time that is worth 1 to 10 % (fewer instructions), except
    // where ptxas then spills: 64 rows at three CTAs per SM, 28 bytes and 6 % slower.
    constexpr bool FULL = VEC && !(TM * TN == 16 && C::CTAS == 3);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int wm = warp % C::WM, wn = warp / C::WM;
    const int nb = K / QBLK;

    // ---- this CTA's unit of work: an output tile (M fastest, so that CTAs running together share weight tiles in L2) and a
    // range of groups [g0, g1); grouped: 128 outputs of one item (up to BM rows of one expert)
    int m0, mend, n0, g0 = 0, g1 = nb, split = 0;
    size_t wrow0 = 0;
    if (GROUPED) {
        const int item = blockIdx.x / n_tiles;
        if (item >= *gl.num_items) return;
        const int4 it = __ldg(gl.items + item);
        m0 = it.y; mend = it.y + it.z; n0 = (blockIdx.x % n_tiles) * BN; wrow0 = (size_t)it.x * N;
    } else {
        const int tiles = m_tiles * n_tiles, tile = blockIdx.x % tiles;
        split = blockIdx.x / tiles;
        m0 = (tile % m_tiles) * BM; mend = M; n0 = (tile / m_tiles) * BN;
        g0 = min(nb, split * gsplit); g1 = min(nb, g0 + gsplit);
    }
    const int nkt = (g1 - g0 + GPK - 1) / GPK;

    // ---- copies: thread -> 16-byte chunk of a row (8 of 128 bytes of activations, 4 of 64 bytes of weights).  Rows past
    // the end are filled with zeros (their scales are the last row's) and never stored; chunks past the last group are skipped.
    constexpr int AI = (BM * 8 + NT - 1) / NT, BI = (BN * 4 + NT - 1) / NT;
    static_assert(BM * 8 % NT == 0 && BN * 4 % NT == 0, "whole copy instructions");
    const uint32_t smem_u = (uint32_t)__cvta_generic_to_shared(smem);
    const int ca = tid & 7, cb = tid & 3;
    const int8_t *Xb = X + (size_t)(m0 + (tid >> 3)) * K + ca * 16;
    const uint8_t *Wb = Wq + (wrow0 + n0 + (tid >> 2)) * (size_t)(K / 2) + cb * 16;
    const int rows_a = mend - m0 - (tid >> 3), rows_b = N - n0 - (tid >> 2);      // live rows from this thread's first one on
    const uint32_t adst = smem_u + (ca >> 1) * C::A_GROUP + (tid >> 3) * 32 + (ca & 1) * 16;
    const uint32_t bdst = smem_u + GPK * C::A_GROUP + cb * C::B_GROUP + (tid >> 2) * 16;
    auto copy = [&](int kt) {
        if (kt < nkt) {
            const int b0 = g0 + kt * GPK, ng = FULL ? GPK : g1 - b0;          // groups left
            const uint32_t so = (uint32_t)(kt % STAGES) * C::STAGE;
            // scales: a row's GPK of them are one 16-byte (fp16: 8-byte) piece when they line up, else 4 bytes at a time.  Ahead of
            // the operands, so that fewer addresses are live at once: 333 x 15360 x 3840, fp16, 163 us, behind them 169.
#pragma unroll
            for (int r = 0; r < C::RA; r++) {
                const int m = tid + r * NT;
                if (BM % NT == 0 || m < BM) {
                    const float *p = xs + (size_t)min(m0 + m, mend - 1) * nb + b0;
                    const uint32_t o = so + C::OFF_SX + m * (GPK * 4);
                    if (VEC) cp_async16(smem_u + o, p, true);
                    else {
#pragma unroll
                        for (int q = 0; q < GPK; q++)
                            if (q < ng) cp_async4(smem_u + o + 4 * q, p + q);
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < C::RB; r++) {
                const int n = tid + r * NT;
                if (BN % NT == 0 || n < BN) {
                    const ST *p = sw + (wrow0 + min(n0 + n, N - 1)) * (size_t)nb + b0;
                    const uint32_t o = so + C::OFF_SW + n * (GPK * 4);
                    if (VEC) {
                        if (sizeof(ST) == 4) cp_async16(smem_u + o, p, true);
                        else cp_async8(smem_u + o, p);
                    } else if (sizeof(ST) == 4 || pairs) {               // pairs: the number of groups is even, so words never straddle the end
                        constexpr int PER = 4 / sizeof(ST);
#pragma unroll
                        for (int q = 0; q < GPK; q += PER)
                            if (q < ng) cp_async4(smem_u + o + sizeof(ST) * q, p + q);
                    } else {
#pragma unroll
                        for (int q = 0; q < GPK; q++)
                            if (q < ng) *reinterpret_cast<ST *>(smem + o + sizeof(ST) * q) = p[q];
                    }
                }
            }
            if ((ca >> 1) < ng) {
                const int8_t *src = Xb + (size_t)b0 * 32;
#pragma unroll
                for (int i = 0; i < AI; i++) {
                    const bool live = i * (NT / 8) < rows_a;
                    cp_async16(adst + so + i * (NT / 8) * 32, live ? src + (size_t)i * (NT / 8) * K : X, live);
                }
            }
            if (cb < ng) {
                const uint8_t *src = Wb + (size_t)b0 * 16;
#pragma unroll
                for (int i = 0; i < BI; i++) {
                    const bool live = i * (NT / 4) < rows_b;
                    cp_async16(bdst + so + i * (NT / 4) * 16, live ? src + (size_t)i * (NT / 4) * (K / 2) : Wq, live);
                }
            }
        }
        cp_async_commit();
    };

    uint64_t acc[TM][TN][2];            // pairs of fp32 sums: row g (columns 2t, 2t + 1), row g + 8
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j][0] = acc[i][j][1] = 0ull;

    const int rows_w = mend - m0 - wm * 16 * TM;                               // live rows of this warp (may be <= 0)
    const int live = GROUPED ? min(TM, (rows_w + 15) / 16) : TM;               // live m16 tiles
    // ng groups of this warp's tile; L = live m16 tiles.  Software pipeline over the columns (n8 tiles) of all groups: the
    // MMAs of the next column are issued before the current one's results are used, because a result takes far longer
    // than the dozen instructions that use it and a warp issues in order.
    auto groups = [&](auto LT, auto NGT, const unsigned char *stage, int bfirst) {
        constexpr int L = decltype(LT)::value, NG = decltype(NGT)::value;
        const unsigned char *As = stage + bfirst * C::A_GROUP + (wm * 16 * TM + g) * 32 + t * 8;
        const unsigned char *Bs = stage + GPK * C::A_GROUP + bfirst * C::B_GROUP + (wn * 8 * TN + g) * 16 + t * 4;
        const unsigned char *sx = stage + C::OFF_SX + (wm * 16 * TM + g) * (GPK * 4) + bfirst * 4;
        const unsigned char *ss = stage + C::OFF_SW + (wn * 8 * TN + 2 * t) * (GPK * 4) + bfirst * sizeof(ST);
        uint32_t a[L][4];
        int c[2][L][4];
        float xx[2][L][2], sv[2][2];
        auto start = [&](int q) {                      // column q % TN of group q / TN: operands, scales, MMAs
            const int bg = q / TN, j = q % TN;
            if (j == 0) {
#pragma unroll
                for (int i = 0; i < L; i++) {
                    const uint2 v0 = *reinterpret_cast<const uint2 *>(As + bg * C::A_GROUP + i * 512), v1 = *reinterpret_cast<const uint2 *>(As + bg * C::A_GROUP + i * 512 + 256);
                    split_even_odd(v0.x, v0.y, a[i][0], a[i][2]);
                    split_even_odd(v1.x, v1.y, a[i][1], a[i][3]);
                    xx[bg & 1][i][0] = *reinterpret_cast<const float *>(sx + bg * 4 + (16 * i) * (GPK * 4));
                    xx[bg & 1][i][1] = *reinterpret_cast<const float *>(sx + bg * 4 + (16 * i + 8) * (GPK * 4));
                }
            }
            uint32_t b0, b1;
            unpack8_x16(*reinterpret_cast<const uint32_t *>(Bs + bg * C::B_GROUP + j * 128), b0, b1);
            sv[q & 1][0] = sval(*reinterpret_cast<const ST *>(ss + bg * sizeof(ST) + 8 * j * (GPK * 4)));
            sv[q & 1][1] = sval(*reinterpret_cast<const ST *>(ss + bg * sizeof(ST) + (8 * j + 1) * (GPK * 4)));
#pragma unroll
            for (int i = 0; i < L; i++) mma_s8(c[q & 1][i], a[i], b0, b1);
        };
        start(0);
#pragma unroll
        for (int q = 0; q < NG * TN; q++) {
            if (q + 1 < NG * TN) start(q + 1);
            const int bg = q / TN, j = q % TN;
            const uint64_t s2 = mul2(pack2(sv[q & 1][0], sv[q & 1][1]), pack2(0.0625f, 0.0625f));
#pragma unroll
            for (int i = 0; i < L; i++) {
                const int (&d)[4] = c[q & 1][i];
                const float x0 = xx[bg & 1][i][0], x1 = xx[bg & 1][i][1];
                fma2(acc[i][j][0], mul2(pack2(__int2float_rn(d[0]), __int2float_rn(d[1])), pack2(x0, x0)), s2);
                fma2(acc[i][j][1], mul2(pack2(__int2float_rn(d[2]), __int2float_rn(d[3])), pack2(x1, x1)), s2);
            }
        }
    };

    // ---- main loop
#pragma unroll
    for (int s = 0; s < STAGES - 1; s++) copy(s);
    for (int kt = 0; kt < nkt; kt++) {
        cp_async_wait<STAGES - 2>();                  // K-tile kt has landed (this thread's copies) ...
        __syncthreads();                              // ... and everybody's; K-tile kt - 1 is done with
        copy(kt + STAGES - 1);                        // into the slot K-tile kt - 1 used
        const unsigned char *stage = smem + (kt % STAGES) * C::STAGE;
        const int ng = FULL ? GPK : min(GPK, g1 - (g0 + kt * GPK));
        auto ktile = [&](auto LT) {
            if (FULL || ng == GPK) groups(LT, std::integral_constant<int, GPK>(), stage, 0);
            else {
#pragma unroll 1
                for (int b = 0; b < ng; b++) groups(LT, std::integral_constant<int, 1>(), stage, b);
            }
        };
        if constexpr (!GROUPED) ktile(std::integral_constant<int, TM>());
        else {                                        // an item's rows rarely fill the tile: only its live m16 tiles cost anything
            if (TM >= 4 && live == 4) ktile(std::integral_constant<int, TM < 4 ? TM : 4>());
            else if (TM >= 3 && live == 3) ktile(std::integral_constant<int, TM < 3 ? TM : 3>());
            else if (TM >= 2 && live == 2) ktile(std::integral_constant<int, TM < 2 ? TM : 2>());
            else if (live == 1) ktile(std::integral_constant<int, 1>());
        }
    }
    cp_async_wait<0>();

    // ---- store: a fragment row is two consecutive columns per lane, four lanes fill a 32-byte sector
    float *Yb = Y + (size_t)split * ((size_t)M * N);
    const bool v2 = ((reinterpret_cast<uintptr_t>(Yb) & 7) == 0) && (N & 1) == 0;
#pragma unroll
    for (int i = 0; i < TM; i++) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int m = m0 + wm * 16 * TM + 16 * i + 8 * h + g;
            if (m < mend) {
                float *yr = Yb + (size_t)m * N;
#pragma unroll
                for (int j = 0; j < TN; j++) {
                    const int n = n0 + wn * 8 * TN + 8 * j + 2 * t;
                    float lo, hi;
                    unpack2(acc[i][j][h], lo, hi);
                    if (v2 && n + 1 < N) *reinterpret_cast<float2 *>(yr + n) = make_float2(lo, hi);
                    else {
                        if (n < N) yr[n] = lo;
                        if (n + 1 < N) yr[n + 1] = hi;
                    }
                }
            }
        }
    }
}

// ---- host side ------------------------------------------------------------------------------------
// A K-tile's scales are one aligned piece of each row.
template <typename ST>
inline bool scales_line_up(const float *xs, const ST *sw, int K, int nsplit, int gsplit) {
    return (K / QBLK) % GPK == 0 && (nsplit == 1 || gsplit % GPK == 0) && aligned(xs, 16) && aligned(sw, 4 * sizeof(ST));
}
// The number of groups and every range of them is even, so that two fp16 scales are one aligned word.
template <typename ST>
inline bool scales_pair_up(const ST *sw, int K, int nsplit, int gsplit) {
    return (K / QBLK) % 2 == 0 && (nsplit == 1 || gsplit % 2 == 0) && aligned(sw, 4);
}
template <class C, typename ST, bool GROUPED, bool VEC>
inline int launch_c(const int8_t *X, const float *xs, const uint8_t *Wq, const ST *sw, float *Y, int M, int N, int K, int nsplit,
                    int gsplit, cudaStream_t st, const GroupList &gl = GroupList(), int max_items = 0) {
    auto kern = gemm_w4a8_mma_kernel<C, ST, GROUPED, VEC>;
    static PerDevice<bool> configured_dev;              // the opt-in is a per-device function attribute
    bool &configured = configured_dev.get();
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
        if (e != cudaSuccess) return cuda_fail(e, "gemm_mma smem opt-in");
        configured = true;
    }
    const int m_tiles = (M + C::BM - 1) / C::BM, n_tiles = (N + C::BN - 1) / C::BN;
    const bool pairs = scales_pair_up(sw, K, nsplit, gsplit);
    const long units = GROUPED ? (long)max_items * n_tiles : (long)m_tiles * n_tiles * nsplit;
    if (units > 0x7FFFFFFFL) return fail(W4A8_ERR_UNSUPPORTED, "gemm: %ld work units", units);
    kern<<<(unsigned)units, C::THREADS, C::SMEM, st>>>(X, xs, Wq, sw, Y, M, N, K, m_tiles, n_tiles, gsplit, pairs, gl);
    return launch_status("gemm_w4a8_mma");
}

using Cfg128 = Cfg<4, 8, 2, 2, 4, 2>;                       // 128 x 128, four warps of 64 x 64, two CTAs per SM
// 16 TM x 128, four warps side by side, three (four) CTAs per SM.  64 rows: three stages instead of four, with which only two
// CTAs would fit (expert block, 128 experts, 512 rows 308 us with four, 283 with three; 128 rows 239 and 204; dense
// 160 x 17408 x 5120 183 and 135).  A grid that leaves one CTA to an SM has nothing but the ring to cover its loads: four.
template <int TM>
using CfgRows = Cfg<TM, 4, 1, 4, TM == 4 ? 3 : 4, TM == 1 ? 4 : 3>;
using Cfg64Deep = Cfg<4, 4, 1, 4, 4, 2>;                    // 112 x 7000 x 3840: 41.1 us, with three stages 43.1

// Which kernel and tile a dense product takes.  The padding of the last row tile, the number of CTAs left over for the last
// wave and the rate of each kind of tile decide; all three follow from the counts and the time a tile needs per group of K
// with 1, 2, 3, 4 of its kind on an SM.  ns: those times, fitted to 13700 timings over M = 8 .. 2048, N = 256 .. 40000 and
// K = 2048 .. 17408, for scales that line up, fp32 scales that are copied 4 bytes at a time, pairs of fp16 scales, and fp16
// scales of an odd K / 32 (plain loads, a latency per K-tile that company on the SM hides).  tcgen05 adds 4 us a wave where N
// is not a multiple of four: its rows are then stored 4 bytes at a time, lane by lane in different rows; 3 us a wave separate it
// from the other kinds' fit for fp32 scales that do not line up.  The sum over waves reproduces the timings to 2 to 8 %.  On
// average over the four the choice is 0.1 to 0.5 % slower than the fastest kind (9 % at most); it is slower than tcgen05 by more than 3 % at one point of the 13700 (65 x 15360 x 2048, 48-row tiles, 4 %).
// Measured, us, chosen kind / tcgen05: 40 x 17408 x 5120 47 / 80, 160 x 17408 x 5120 131 / 166, 333 x 15360 x 3840 158 / 187,
// 512 x 17408 x 5120 296 / 327, 24 x 20000 x 4128 53 / 122; tcgen05 / 64 rows: 700 x 9000 x 5024 240 / 254, 128 x 17408 x 5120
// 87 / 91.  16 and 32 rows were not timed above max_rows.  128 x 128 tiles with scales 4 bytes at a time were never the fastest
// kind for fp32 scales and at most 7 % ahead for fp16, so there are none.
enum class Tile { TC, T128, R16, R32, R48, R64 };
enum Scales { LINED_UP, WORDS, PAIRS, HALVES };
inline Tile pick(long M, long N, int K, int nsplit, int gsplit, Scales scales) {
    struct Kind { Tile tile; int rows, per_sm; long ns[4][4], max_rows; };
    static const Kind kinds[6] = {
        {Tile::TC, 128, 1, {{485}, {475}, {560}, {570}}, 1L << 31},
        {Tile::T128, 128, 2, {{510, 935}, {0}, {0}, {0}}, 1L << 31},
        {Tile::R16, 16, 4, {{155, 295, 470, 630}, {180, 435, 555, 720}, {175, 390, 480, 640}, {350, 475, 655, 850}}, 16},
        {Tile::R32, 32, 3, {{200, 375, 525}, {225, 390, 530}, {220, 370, 515}, {405, 510, 600}}, 128},
        {Tile::R48, 48, 3, {{255, 460, 635}, {275, 490, 725}, {260, 500, 690}, {410, 585, 735}}, 1L << 31},
        {Tile::R64, 64, 3, {{295, 535, 760}, {320, 545, 795}, {315, 545, 790}, {430, 625, 820}}, 1L << 31}};
    const long sms = sm_count(), n_tiles = (N + 127) / 128 * nsplit, groups = nsplit > 1 ? gsplit : K / QBLK;
    Tile best = Tile::TC;
    long best_ns = 0;
    for (const Kind &k : kinds) {
        const long *ns = k.ns[scales];
        if (M > k.max_rows || ns[0] == 0) continue;
        const long ctas = (M + k.rows - 1) / k.rows * n_tiles, wave = sms * k.per_sm, rest = ctas % wave;
        long t = (ctas / wave * ns[k.per_sm - 1] + (rest ? ns[(rest + sms - 1) / sms - 1] : 0)) * groups;
        if (k.tile == Tile::TC) t += (ctas + sms - 1) / sms * ((scales == WORDS ? 3000 : 0) + (N % 4 != 0 ? 4000 : 0));
        if (best_ns == 0 || t < best_ns) { best = k.tile; best_ns = t; }
    }
    return best;
}

template <typename ST>
inline int launch_t(const int8_t *X, const float *xs, const uint8_t *Wq, const ST *sw, float *Y, int M, int N, int K, int nsplit,
                    int gsplit, cudaStream_t st) {
    const bool lines_up = scales_line_up(xs, sw, K, nsplit, gsplit);
    const Scales scales = lines_up ? LINED_UP : sizeof(ST) == 4 ? WORDS : scales_pair_up(sw, K, nsplit, gsplit) ? PAIRS : HALVES;
    const auto run = [&](auto c) {
        using C = decltype(c);
        if (lines_up) return launch_c<C, ST, false, true>(X, xs, Wq, sw, Y, M, N, K, nsplit, gsplit, st);
        return launch_c<C, ST, false, false>(X, xs, Wq, sw, Y, M, N, K, nsplit, gsplit, st);
    };
    switch (pick(M, N, K, nsplit, gsplit, scales)) {
        case Tile::T128: return launch_c<Cfg128, ST, false, true>(X, xs, Wq, sw, Y, M, N, K, nsplit, gsplit, st);
        case Tile::R16: return run(CfgRows<1>());
        case Tile::R32: return run(CfgRows<2>());
        case Tile::R48: return run(CfgRows<3>());
        case Tile::R64:
            if (lines_up && (long)((M + 63) / 64) * ((N + 127) / 128) * nsplit <= sm_count())
                return launch_c<Cfg64Deep, ST, false, true>(X, xs, Wq, sw, Y, M, N, K, nsplit, gsplit, st);
            return run(CfgRows<4>());
        case Tile::TC: break;
    }
    return gemm::launch_tc_t<ST, false>(X, xs, Wq, sw, Y, nullptr, M, N, K, nsplit, gsplit, st, OutArgs());
}

// nsplit = 1: Y is the output.  nsplit > 1: Y is the [nsplit][M][N] partial-sum workspace and gsplit the number of groups
// per split (a split without groups stores zeros).  X and Wq 16-byte aligned; the caller checks.
inline int launch(const int8_t *X, const float *xs, const uint8_t *Wq, const void *sw, float *Y, int M, int N, int K, int scale_dtype,
                  int nsplit, int gsplit, cudaStream_t st) {
    if (scale_dtype == 1) return launch_t<__half>(X, xs, Wq, (const __half *)sw, Y, M, N, K, nsplit, gsplit, st);
    return launch_t<float>(X, xs, Wq, (const float *)sw, Y, M, N, K, nsplit, gsplit, st);
}

// Grouped experts: Y[sorted row, n] for the rows and experts the item list names (rows no item covers are not written).
inline int launch_grouped(const int8_t *X, const float *xs, const uint8_t *Wq, const void *sw, float *Y, int rows, int N, int K,
                          int scale_dtype, const GroupList &gl, int max_items, cudaStream_t st) {
    using C = CfgRows<4>;
    static_assert(C::BM == ITEM_ROWS, "an item's rows are one tile");
    const int gsplit = K / QBLK;
    const auto run = [&](auto *w) {
        using ST = std::remove_const_t<std::remove_pointer_t<decltype(w)>>;
        if (scales_line_up(xs, w, K, 1, gsplit)) return launch_c<C, ST, true, true>(X, xs, Wq, w, Y, rows, N, K, 1, gsplit, st, gl, max_items);
        return launch_c<C, ST, true, false>(X, xs, Wq, w, Y, rows, N, K, 1, gsplit, st, gl, max_items);
    };
    return scale_dtype == 1 ? run((const __half *)sw) : run((const float *)sw);
}

}  // namespace gemm_mma
}  // namespace w4a8
