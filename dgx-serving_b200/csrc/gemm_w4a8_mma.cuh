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
// Alone (a loop without loads) MMA 270, I2F 256 (on the ALU pipe) and packed mul + fma 278 cycles per 128 x 128 group; together
// 630, because the legacy tensor path and the packed fp32 pipe take turns: that is the floor of this kernel.  At 1965 MHz it needs
// 750 at 2048 x 17408 x 5120 (two CTAs of 80 rows per SM), 880 at 333 x 15360 x 3840 (three of 48) and about 1100 where an SM has one
// CTA of 48: it has one warp per scheduler, and nothing covers its waits.  Measured, us, with the quantizer, with cp.async operands /
// with TMA / with the shorter unpacking and the later start as well: these two 1088 / 942 / 913 and 164 / 123 / 119, 48 x 3840 x 15360
// in three K ranges, twice, 106 / 86 / 80.  Slower in the first versions, in cycles per 128 x 128 group: integer-to-float through a preset accumulator (1.5 * 2^23)
// instead of I2F (1133 against 989), scalar instead of packed fp32 (1044 against 864), scales through registers (977 against 864;
// they spill).  Thin tiles with cp.async operands, 32 x 3840 x 15360 in three ranges: 41 us; 8 and 16 warps per CTA 45 and 49,
// K-tiles of 8 groups 43, rows prefetched to L2 47 to 61.  A barrier asked ahead of time, so that a CTA does not wait for the answer:
// 2 % with one CTA per SM, but the CTAs of an SM then keep step and those of a last wave pair up (1208 x 3189 x 3840 98 / 119).
//
// Data flow.  TMA brings K-tiles of 4 groups into a STAGES-deep ring, one barrier per stage: activations in the 128-byte swizzle
// (a row's 4 groups), packed weights in the 64-byte one.  With cp.async the same copies, 16 bytes a lane, ran at 13 bytes per cycle
// and SM and took the issue slots of the warps that multiply: without any copies 333 x 15360 x 3840 then took 119 us instead of 164.
// Fragment reads are contiguous up to the swizzle (LDS.64 and LDS.32, no conflicts).  A lane's word of weights expands to its two B
// registers with three logic operations (unpack8_x16: even and odd elements), the matching A registers are two byte permutes of
// eight activations.  Any order of K inside a group gives the same integer.  Scales travel with their K-tile by cp.async,
// [row][group], one 16-byte (fp16: 8-byte) piece per row where they line up, that is where K / 32 and every range of a split K are
// multiples of four and the pointers aligned (VEC); 4 bytes at a time otherwise, and fp16 scales of an odd K / 32, whose rows start
// between two words, by plain loads, which stall their warp once per K-tile.  One __syncthreads per K-tile; two or three CTAs per SM
// cover each other.
#pragma once
#include <cuda.h>
#include <type_traits>
#include "common.cuh"
#include "gemm_w4a8_tc.cuh"
#include "tma_ring.cuh"

namespace w4a8 {
namespace gemm_mma {

constexpr int GPK = 4;                    // groups per K-tile
constexpr unsigned SMS = 148;             // of a B200: the first 148 CTAs of a launch are on an SM each, the next 148 beside them
// bytes = 0 writes zeros and reads nothing
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
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
    static constexpr int A_STAGE = BM * GPK * 32, B_STAGE = BN * GPK * 16;
    static constexpr int OFF_SX = A_STAGE + B_STAGE, OFF_SW = OFF_SX + BM * GPK * 4;      // scales: [row][group]
    static constexpr int STAGE = (OFF_SW + BN * GPK * 4 + 1023) / 1024 * 1024;            // the swizzle repeats every 1024 bytes
    static constexpr int OFF_BAR = STAGES * STAGE, SMEM = OFF_BAR + STAGES * 8;
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
    long likely_items = 0;                                 // what the host expects, for the form of the launch only
};

template <class C, typename ST, bool GROUPED, bool VEC>
__global__ void __launch_bounds__(C::THREADS, C::CTAS) gemm_w4a8_mma_kernel(
    const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const float *__restrict__ xs, const ST *__restrict__ sw,
    float *__restrict__ Y, int M, int N, int K, int m_tiles, int n_tiles, int gsplit, bool pairs, int stagger, const GroupList gl) {
    extern __shared__ __align__(1024) unsigned char smem[];
    constexpr int TM = C::TM, TN = C::TN, BM = C::BM, BN = C::BN, NT = C::THREADS, STAGES = C::STAGES;
    constexpr bool FULL = VEC;                             // scales that line up make every K-tile complete: 1 to 10 % faster when known here
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int wm = warp % C::WM, wn = warp / C::WM;
    const int nb = K / QBLK;

    // ---- this CTA's unit of work: an output tile (M fastest, so that CTAs running together share weight tiles in L2) and a
    // range of groups [g0, g1); grouped: 128 outputs of one item (up to BM rows of one expert)
    int m0, mend, n0, g0 = 0, g1 = nb, split = 0;
    size_t wrow0 = 0;
    if (GROUPED) {
        pdl_wait();                                        // the items and the rows come from the kernel before this one
        pdl_launch_dependents();
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

    // ---- copies.  Rows and columns past the end come from the next expert or are zeros, and are never stored.
    // The thread that starts the bulk copies.  Where one warp copies all of the activations' scales besides, it is one of the last
    // warp: 16 x 18944 x 5120 24.8 us by the first thread, 23.1 so; 192 x 9472 x 5120 56.6 and 59.1.
    constexpr int ISSUER = !GROUPED && BM <= 32 ? NT - 32 : 0;
    const uint32_t smem_u = (uint32_t)__cvta_generic_to_shared(smem);
    auto FULL_BAR = [&](int i) { return smem_u + C::OFF_BAR + 8u * i; };
    // The second CTA of an SM starts `stagger` cycles after the first (host side: stagger_cycles).
    if (C::CTAS == 2 && !GROUPED && stagger > 0 && blockIdx.x < 2 * SMS && blockIdx.x >= SMS) {
        const long long t1 = clock64() + stagger;
        while (clock64() < t1) __nanosleep(200);
    }
    if (tid == 0) {
        for (int i = 0; i < STAGES; i++) ptx::mbar_init(FULL_BAR(i), 1);
        ptx::mbar_fence_init();
        ptx::tma_prefetch_desc(&tmX);
        ptx::tma_prefetch_desc(&tmW);
    }
    __syncthreads();
    static_assert(!GROUPED || C::WM == 1, "an item's live tiles are every warp's");
    const int live = GROUPED ? min(TM, (mend - m0 + 15) / 16) : TM;            // live m16 tiles
    // Scales past the end: the address is the last row's, the 16-byte copies (which pass L1 by) read nothing from it.  When they did,
    // all lanes past the end of all CTAs of a column, or of all CTAs with few rows, asked L2 for the same 16 bytes:
    // 2034 x 162 x 5376 67.6 us, 30.7 so; one row x 18944 x 5120 29.4, 22.7 so.
    int bytes_a[C::RA], bytes_b[C::RB];
#pragma unroll
    for (int r = 0; r < C::RA; r++) bytes_a[r] = m0 + tid + r * NT < mend ? 16 : 0;
#pragma unroll
    for (int r = 0; r < C::RB; r++) bytes_b[r] = n0 + tid + r * NT < N ? 16 : 0;
    auto copy = [&](int kt, bool ok) {
        if (kt < nkt) {
            const int b0 = g0 + kt * GPK, ng = FULL ? GPK : g1 - b0;          // groups left
            const uint32_t so = (uint32_t)(kt % STAGES) * C::STAGE;
            if (tid == ISSUER && ok) {
                if (GROUPED) {                                                // only the item's live m16 tiles, 16 rows a copy
                    ptx::mbar_arrive_expect_tx(FULL_BAR(kt % STAGES), live * 2048 + C::B_STAGE);
                    for (int i = 0; i < live; i++) ptx::tma_load_2d(smem_u + so + i * 2048, &tmX, b0 * 32, m0 + 16 * i, FULL_BAR(kt % STAGES));
                } else {
                    ptx::mbar_arrive_expect_tx(FULL_BAR(kt % STAGES), C::A_STAGE + C::B_STAGE);
                    ptx::tma_load_2d(smem_u + so, &tmX, b0 * 32, m0, FULL_BAR(kt % STAGES));
                }
                ptx::tma_load_2d(smem_u + so + C::A_STAGE, &tmW, b0 * 16, (int)wrow0 + n0, FULL_BAR(kt % STAGES));
            }
            // scales: a row's GPK of them are one 16-byte (fp16: 8-byte) piece when they line up, else 4 bytes at a time, neighbours by
            // neighbouring lanes, so that an instruction touches 8 (pairs: 16) rows and not 32: 4 x 5004 x 4192 27.8 us with a row
            // per lane, 21.3 so; 300 x 9000 x 4128 fp32 107.5 and 99.8, fp16 118 and 104
            if (VEC) {
#pragma unroll
                for (int r = 0; r < C::RA; r++) {
                    const int m = tid + r * NT;
                    if (BM % NT == 0 || m < BM) cp_async16(smem_u + so + C::OFF_SX + m * (GPK * 4), xs + (size_t)min(m0 + m, mend - 1) * nb + b0, bytes_a[r]);
                }
#pragma unroll
                for (int r = 0; r < C::RB; r++) {
                    const int n = tid + r * NT;
                    if (BN % NT == 0 || n < BN) {
                        const ST *p = sw + (wrow0 + min(n0 + n, N - 1)) * (size_t)nb + b0;
                        if (sizeof(ST) == 4) cp_async16(smem_u + so + C::OFF_SW + n * (GPK * 4), p, bytes_b[r]);
                        else cp_async8(smem_u + so + C::OFF_SW + n * (GPK * 4), p);
                    }
                }
            } else {
                const int q = tid % GPK;
                if (q < ng) {
#pragma unroll
                    for (int m = tid / GPK; m < BM; m += NT / GPK)
                        cp_async4(smem_u + so + C::OFF_SX + (m * GPK + q) * 4, xs + (size_t)min(m0 + m, mend - 1) * nb + b0 + q);
                }
                auto row = [&](int n) { return sw + (wrow0 + min(n0 + n, N - 1)) * (size_t)nb + b0; };
                if (sizeof(ST) == 2 && pairs) {                          // the number of groups is even, so words never straddle the end
                    const int h = tid % (GPK / 2) * 2;
                    if (h < ng) {
#pragma unroll
                        for (int n = tid / (GPK / 2); n < BN; n += NT / (GPK / 2)) cp_async4(smem_u + so + C::OFF_SW + n * (GPK * 4) + h * 2, row(n) + h);
                    }
                } else if (q < ng) {
#pragma unroll
                    for (int n = tid / GPK; n < BN; n += NT / GPK) {
                        if (sizeof(ST) == 4) cp_async4(smem_u + so + C::OFF_SW + (n * GPK + q) * 4, row(n) + q);
                        else *reinterpret_cast<ST *>(smem + so + C::OFF_SW + n * (GPK * 4) + q * 2) = row(n)[q];
                    }
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

    // Fragment row g is row gr of its eight: with it the eight-byte reads of half a warp (g = 0..3) meet four different pairs of
    // swizzled chunks.
    const int gr = ((g & 3) << 1) | (g >> 2);
    const uint32_t aoff = gr * 128 + (((t >> 1) ^ gr) << 4) + (t & 1) * 8, boff = g * 64 + ((g >> 1) << 4) + t * 4;
    // ng groups of this warp's tile; L = live m16 tiles.  Software pipeline over the columns (n8 tiles) of all groups: the
    // MMAs of the next column are issued before the current one's results are used, because a result takes far longer
    // than the dozen instructions that use it and a warp issues in order.
    auto groups = [&](auto LT, auto NGT, const unsigned char *stage, int bfirst) {
        constexpr int L = decltype(LT)::value, NG = decltype(NGT)::value;
        const unsigned char *As = stage + (wm * 16 * TM) * 128, *Bs = stage + C::A_STAGE + (wn * 8 * TN) * 64;
        const unsigned char *sx = stage + C::OFF_SX + (wm * 16 * TM + gr) * (GPK * 4) + bfirst * 4;
        const unsigned char *ss = stage + C::OFF_SW + (wn * 8 * TN + 2 * t) * (GPK * 4) + bfirst * sizeof(ST);
        // the swizzles put chunk c of a row where c ^ (row & 7) (activations) and c ^ (row / 2 & 3) (weights) would be: for group b
        // that is an exclusive or with b on the lane's offset for group 0
        uint32_t a[L][4];
        int c[2][L][4];
        float xx[2][L][2], sv[2][2];
        auto start = [&](int q) {                      // column q % TN of group q / TN: operands, scales, MMAs
            const int bg = q / TN, j = q % TN;
            if (j == 0) {
#pragma unroll
                for (int i = 0; i < L; i++) {
                    const unsigned char *pa = As + (aoff ^ ((bfirst + bg) << 5)) + i * 2048;
                    const uint2 v0 = *reinterpret_cast<const uint2 *>(pa), v1 = *reinterpret_cast<const uint2 *>(pa + 1024);
                    split_even_odd(v0.x, v0.y, a[i][0], a[i][2]);
                    split_even_odd(v1.x, v1.y, a[i][1], a[i][3]);
                    xx[bg & 1][i][0] = *reinterpret_cast<const float *>(sx + bg * 4 + (16 * i) * (GPK * 4));
                    xx[bg & 1][i][1] = *reinterpret_cast<const float *>(sx + bg * 4 + (16 * i + 8) * (GPK * 4));
                }
            }
            uint32_t b0, b1;
            // Two tiles that the shorter form of the unpacking slows down, timed on the shapes that take them with the second CTA of an SM
            // starting later: time of the longer form over the shorter one, 64 rows with fp32 scales 0.97 (scales that do not line up 1.00,
            // and steadier), 80 rows with fp16 scales that line up 0.995, that do not 1.02; 32 and 48 rows 1.01 to 1.03, 64 rows fp16 1.04,
            // 80 rows fp32 1.02, 96 rows 1.02 to 1.03.
            constexpr bool EXPR = !GROUPED && ((TM == 4 && sizeof(ST) == 4) || (TM == 5 && sizeof(ST) == 2 && VEC));
            const uint32_t word = *reinterpret_cast<const uint32_t *>(Bs + (boff ^ ((bfirst + bg) << 4)) + j * 512);
            if constexpr (EXPR) unpack8_x16_expr(word, b0, b1);
            else unpack8_x16(word, b0, b1);
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
    auto landed = [&](int kt) { return ptx::mbar_wait(FULL_BAR(kt % STAGES), (uint32_t)(kt / STAGES) & 1u); };
    auto sync = [&](int) {
        cp_async_wait<STAGES - 2>();                  // this thread's scales; everybody's behind the barrier
        __syncthreads();
    };
    auto use = [&](int kt) {
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
    };
    auto settle = [&]() {
        dev_set_error(0x600u);                        // the outputs are void
        const long long t0 = clock64();
        while (clock64() - t0 < (1ll << 21)) { }
    };
    run_ring<STAGES>(nkt, copy, landed, sync, use, settle);
    cp_async_wait<0>();

    // ---- store: a fragment row is two consecutive columns per lane, four lanes fill a 32-byte sector
    float *Yb = Y + (size_t)split * ((size_t)M * N);
    const bool v2 = ((reinterpret_cast<uintptr_t>(Yb) & 7) == 0) && (N & 1) == 0;
#pragma unroll
    for (int i = 0; i < TM; i++) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int m = m0 + wm * 16 * TM + 16 * i + 8 * h + gr;
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
// Two CTAs of an SM that start together end together, and those of the last wave then pair up on the SMs that come free first; they
// also want the same pipes at the same time.  So where there is more than one wave the second CTA of an SM starts later: 5 % of a tile's
// time, which is about what SMs differ by, or 12 % where the last wave has at most one CTA per SM and pairing up costs most.  Time over
// that without, 0 / 3 / 5 / 8 / 12 %, mean over the shapes of 17967 random ones: last wave of at most one CTA per SM behind one full
// wave, 64 rows 1 / 0.92 / 0.88 / 0.86 / 0.85, 80 rows 1 / 0.87 / 0.84 / 0.83 / 0.83 (and the worst twentieth of them 1.00 of the time
// before the shorter unpacking, 1.12 with 5 %), behind two 80 rows 1 / 0.96 / 0.95 / 0.94 / 0.93; larger last waves, 80 rows
// 1 / 1.00 / 1.00 / 1.00 / 1.01.  96 rows with fp32 scales that line up gain nothing from more than 5 %: 1 / 0.93 / 0.92 / 0.93 / 0.94.
// Three and four CTAs per SM drift apart by themselves (48 rows: 154.8 / 155.1; 333 x 15360 x 3840 116 / 118).  Not on a chip whose
// number of SMs is another one.
inline int stagger_cycles(long ctas, int per_sm, int rows, int groups, bool more) {
    if (per_sm != 2 || sm_count() != (int)SMS || ctas <= 2 * (long)SMS) return 0;
    const long rest = ctas % (2 * (long)SMS);
    const long cycles = (long)groups * rows * 12 * (more && rest > 0 && rest <= (long)SMS ? 12 : 5) / 100;  // a group of a tile's row takes about 12 with two CTAs on the SM
    return (int)(cycles < 100000 ? cycles : 100000);
}
template <class C, typename ST, bool GROUPED, bool VEC>
inline int launch_c(const int8_t *X, const float *xs, const uint8_t *Wq, const ST *sw, float *Y, int M, int N, int K, int nsplit,
                    int gsplit, cudaStream_t st, const GroupList &gl = GroupList(), int max_items = 0, long w_rows = 0) {
    CUtensorMap tmX, tmW;
    int rc = make_tmap_u8(&tmX, X, (uint64_t)K, (uint64_t)M, GPK * 32, GROUPED ? 16 : C::BM, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc == W4A8_OK) rc = make_tmap_u8(&tmW, Wq, (uint64_t)K / 2, (uint64_t)(GROUPED ? w_rows : N), GPK * 16, C::BN, CU_TENSOR_MAP_SWIZZLE_64B);
    if (rc != W4A8_OK) return rc;
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
    // Grouped: dependent where the items fill the SMs.  With fewer units than two per SM the CTAs that start early pair up beside what is
    // still running.  Expert block, us, dependent / not: 94 tokens, 16 experts, 8 of them, 1024 x 512 (128 units) 37.2 / 30.5;
    // 21, 8, 8, 2048 x 768 (96, 128) 38.0 / 31.6; 362, 32, 4, 512 x 1024 (512, 128) 47.1 / 43.5; 176, 8, 8, 1024 x 512 (192) 40.7 / 39.7;
    // 300, 16, 8, 1024 x 512 (384) 60.4 / 61.1; 400, 64, 2, 1024 x 512 (512) 41.0 / 41.9; 20, 64, 8, 2048 x 768 (768) 80.8 / 81.5.
    const bool dependent = GROUPED && gl.likely_items * n_tiles > 2L * sm_count();
    const int stagger = GROUPED ? 0 : stagger_cycles(units, C::CTAS, C::BM, nsplit > 1 ? gsplit : K / QBLK, !(C::BM == 96 && sizeof(ST) == 4 && VEC));
    if (dependent) {
        const cudaError_t e = launch_pdl(kern, dim3((unsigned)units), dim3(C::THREADS), C::SMEM, st, tmX, tmW, xs, sw, Y, M, N, K, m_tiles, n_tiles, gsplit, pairs, stagger, gl);
        if (e != cudaSuccess) return cuda_fail(e, "gemm_w4a8_mma launch");
    } else kern<<<(unsigned)units, C::THREADS, C::SMEM, st>>>(tmX, tmW, xs, sw, Y, M, N, K, m_tiles, n_tiles, gsplit, pairs, stagger, gl);
    return launch_status("gemm_w4a8_mma");
}

// Rows of a tile / CTAs per SM; 128 columns, four warps side by side.  64 rows at two CTAs or three: the deeper ring, or the fuller
// last wave; three with fp32 scales would spill.
using Cfg16 = Cfg<1, 4, 1, 4, 4, 4>;
using Cfg32 = Cfg<2, 4, 1, 4, 4, 3>;
using Cfg48 = Cfg<3, 4, 1, 4, 4, 3>;
using Cfg64 = Cfg<4, 4, 1, 4, 4, 2>;
using Cfg64x3 = Cfg<4, 4, 1, 4, 3, 3>;
using Cfg80 = Cfg<5, 4, 1, 4, 4, 2>;
using Cfg96 = Cfg<6, 4, 1, 4, 4, 2>;

// Which tile a dense product takes.  The padding of the last row tile, the number of CTAs left over for the last wave and the rate
// of each kind of tile decide; all three follow from the counts and from times of the tile.  wave_ns: what a wave takes apart from
// K.  ns: a group of K with 1, 2, 3, 4 of its kind on an SM.  tail_ns: the same in a wave behind full ones, which starts as slots
// come free.  Five columns each: fp32 scales that line up, fp32 scales copied 4 bytes at a time, pairs of fp16 scales, fp16 scales
// of an odd K / 32 (plain loads), fp16 scales that line up.  Fitted to 16874 shapes, M = 1 .. 2048, N = 64 .. 20000, one to eight
// ranges of 1 to 200 groups, on which every tile was timed, with the longer unpacking and no later start.  With both as they are now, on
// 9482 other shapes of these ranges: the choice is 0.6 to 0.8 % slower than the fastest tile on average, 10 to 12 % at the 99th
// percentile.  A tile taller than one that holds all rows has only more padding; 16 rows were not timed above
// max_rows.  Not among them because never or hardly ever ahead: 128 x 128 tiles (fastest for 32 of 15284 shapes, by a few per cent)
// and the tcgen05 kernel (for none).
enum class Tile { R16, R32, R48, R64, R64X3, R80, R96 };
enum Scales { LINED_UP, WORDS, PAIRS, HALVES, LINED_UP_FP16 };
inline Tile pick(long M, long N, int K, int nsplit, int gsplit, Scales scales) {
    constexpr long ANY = 1L << 31;
    struct Kind { Tile tile; int rows, per_sm; long max_rows, wave_ns[5], ns[5][4], tail_ns[5][3]; };
    static const Kind kinds[] = {
        {Tile::R16, 16, 4, 160, {1935, 1885, 1970, 2110, 1840},
         {{125, 235, 320, 350}, {145, 265, 365, 390}, {155, 250, 345, 380}, {185, 280, 360, 425}, {130, 235, 340, 370}},
         {{70, 150, 205}, {75, 165, 275}, {55, 125, 180}, {75, 145, 260}, {30, 125, 200}}},
        {Tile::R32, 32, 3, ANY, {2255, 2175, 2250, 2520, 2140},
         {{170, 330, 360}, {190, 325, 380}, {195, 315, 370}, {215, 340, 390}, {170, 310, 345}},
         {{160, 280}, {170, 300}, {110, 260}, {145, 295}, {105, 240}}},
        {Tile::R48, 48, 3, ANY, {2755, 2635, 2725, 2985, 2640},
         {{205, 390, 490}, {230, 445, 530}, {240, 410, 510}, {260, 430, 540}, {200, 395, 485}},
         {{170, 330}, {175, 365}, {190, 345}, {170, 375}, {170, 335}}},
        {Tile::R64, 64, 2, ANY, {2935, 2745, 2815, 3130, 2825},
         {{255, 425}, {270, 450}, {290, 445}, {305, 475}, {255, 420}},
         {{225}, {285}, {310}, {285}, {275}}},
        {Tile::R64X3, 64, 3, ANY, {0, 0, 3095, 3520, 3075},
         {{0}, {0}, {285, 480, 655}, {300, 490, 660}, {250, 475, 635}},
         {{0}, {0}, {130, 425}, {245, 425}, {145, 415}}},
        {Tile::R80, 80, 2, ANY, {3450, 3180, 3220, 3635, 3355},
         {{290, 505}, {345, 520}, {355, 530}, {365, 555}, {290, 485}},
         {{260}, {390}, {405}, {445}, {355}}},
        {Tile::R96, 96, 2, ANY, {4080, 3415, 3490, 4075, 3930},
         {{365, 595}, {400, 610}, {390, 600}, {400, 635}, {360, 575}},
         {{305}, {400}, {445}, {495}, {420}}}};
    const long sms = sm_count(), n_tiles = (N + 127) / 128 * nsplit, groups = nsplit > 1 ? gsplit : K / QBLK;
    Tile best = Tile::R16;
    long best_ns = 0;
    int holds_all = 0;                                      // rows of the shortest tile that holds all rows
    for (const Kind &k : kinds) {
        if (M > k.max_rows || k.wave_ns[scales] == 0) continue;
        if (holds_all && k.rows > holds_all) break;
        if (k.rows >= M) holds_all = k.rows;
        const long ctas = (M + k.rows - 1) / k.rows * n_tiles, wave = sms * k.per_sm, full = ctas / wave, rest = ctas % wave;
        const long last = (rest + sms - 1) / sms;           // CTAs per SM in the last wave
        const long last_ns = last == 0 ? 0 : full == 0 || last == k.per_sm ? k.ns[scales][last - 1] : k.tail_ns[scales][last - 1];
        long t = (full + (last != 0)) * k.wave_ns[scales] + (full * k.ns[scales][k.per_sm - 1] + last_ns) * groups;
        // 96 rows whose last wave behind a full one pairs up now and then whatever the later start: 801 x 6272 x 3968 141 us, 118 in 48 rows
        if (k.tile == Tile::R96 && scales == LINED_UP && full == 1 && last == 1) t += t / 20;
        if (best_ns == 0 || t < best_ns) { best = k.tile; best_ns = t; }
    }
    return best;
}

template <typename ST>
inline int launch_t(const int8_t *X, const float *xs, const uint8_t *Wq, const ST *sw, float *Y, int M, int N, int K, int nsplit,
                    int gsplit, cudaStream_t st) {
    const bool lines_up = scales_line_up(xs, sw, K, nsplit, gsplit);
    const Scales scales = lines_up ? (sizeof(ST) == 4 ? LINED_UP : LINED_UP_FP16) : sizeof(ST) == 4 ? WORDS : scales_pair_up(sw, K, nsplit, gsplit) ? PAIRS : HALVES;
    const auto run = [&](auto c) {
        using C = decltype(c);
        if (lines_up) return launch_c<C, ST, false, true>(X, xs, Wq, sw, Y, M, N, K, nsplit, gsplit, st);
        return launch_c<C, ST, false, false>(X, xs, Wq, sw, Y, M, N, K, nsplit, gsplit, st);
    };
    switch (pick(M, N, K, nsplit, gsplit, scales)) {
        case Tile::R16: return run(Cfg16());
        case Tile::R32: return run(Cfg32());
        case Tile::R48: return run(Cfg48());
        case Tile::R64: return run(Cfg64());
        case Tile::R64X3:
            if constexpr (sizeof(ST) == 2) return run(Cfg64x3());
            break;
        case Tile::R80: return run(Cfg80());
        case Tile::R96: break;
    }
    return run(Cfg96());
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
                          int scale_dtype, const GroupList &gl, int max_items, long w_rows, cudaStream_t st) {
    using C = Cfg64;            // expert block, 128 experts, 512 rows: 244 us; three CTAs of three stages, which spill, 302
    static_assert(C::BM == ITEM_ROWS, "an item's rows are one tile");
    const int gsplit = K / QBLK;
    const auto run = [&](auto *w) {
        using ST = std::remove_const_t<std::remove_pointer_t<decltype(w)>>;
        if (scales_line_up(xs, w, K, 1, gsplit)) return launch_c<C, ST, true, true>(X, xs, Wq, w, Y, rows, N, K, 1, gsplit, st, gl, max_items, w_rows);
        return launch_c<C, ST, true, false>(X, xs, Wq, w, Y, rows, N, K, 1, gsplit, st, gl, max_items, w_rows);
    };
    return scale_dtype == 1 ? run((const __half *)sw) : run((const float *)sw);
}

}  // namespace gemm_mma
}  // namespace w4a8
