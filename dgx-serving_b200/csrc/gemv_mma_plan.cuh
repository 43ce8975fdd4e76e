// Shared-memory plan of the tensor-path GEMV (gemv_w4a8_mma.cuh): how many groups a step has, how deep the rings are, whether tiles are
// relayed.  No CUDA construct in it beyond the qualifiers, so that the same text is checked on the CPU over all sizes.
#pragma once
#include <cstddef>
#ifdef __CUDACC__
#define W4A8_PLAN_FN __host__ __device__ constexpr
#else
#define W4A8_PLAN_FN constexpr
#endif

namespace w4a8 {
namespace gemv_mma {

#ifndef W4A8_MMA_WARPS
#define W4A8_MMA_WARPS 8
#endif
constexpr int WARPS = W4A8_MMA_WARPS;
#ifndef W4A8_GEMV_RELAY
#define W4A8_GEMV_RELAY 1
#endif
constexpr bool RELAY = W4A8_GEMV_RELAY != 0;
constexpr int RELAY16_TILES = 2;                 // 9 to 16 rows: most 16-row tiles of a CTA that are relayed
// A step = 16 weight rows x GS groups (GS * 16 B contiguous per row) plus the 16 x GS scales (slot sized for fp32).
W4A8_PLAN_FN int step_w(int GS) { return 16 * GS * 16; }
W4A8_PLAN_FN int step_bytes(int GS) { return 16 * GS * 16 + 16 * GS * 4; }

// Dynamic shared memory (bytes), all offsets multiples of 16; MH = 1 for up to eight rows, 2 for up to sixteen:
//   xq'  : S rows x pitch2 uint2      (pitch2 = 4*nb + 4: rows 4 uint2 apart modulo 16 -> conflict-free LDS.64)
//   xs'  : nb x (8*MH) floats          ([group][m], already multiplied by 1/16)
//   ring : WARPS x STAGES x step_bytes(GS)
// Only the S rows that exist are staged, so a single-row decode call keeps its footprint small enough for the next kernel's CTA to
// become resident beside it; the MMA's columns from S on repeat the last row and are never stored.
W4A8_PLAN_FN int pitch2_of(int nb) { return 4 * nb + 4; }
W4A8_PLAN_FN size_t xq_bytes(int S, int nb) { return (size_t)S * pitch2_of(nb) * 8; }
W4A8_PLAN_FN size_t act_bytes(int MH, int S, int nb) { return xq_bytes(S, nb) + (size_t)nb * 8 * MH * 4; }
W4A8_PLAN_FN size_t smem_bytes(int MH, int S, int nb, int GS, int STAGES) {
    return act_bytes(MH, S, nb) + (size_t)WARPS * STAGES * step_bytes(GS);
}
// Static shared memory of the kernel: the relay's mailboxes and flags, or what the peer form needs to publish; rounded up to 1 KB, the
// alignment that the dynamic part has in this library.
W4A8_PLAN_FN size_t static_bytes(int MH, bool relay) {
    return relay ? ((size_t)(WARPS / 2) * (MH * 512 + 4) + 64 + 1023) / 1024 * 1024 : 1024;
}
constexpr size_t SMEM_CTA = 227 * 1024;          // of an SM's shared memory, what one CTA may have, static and dynamic
constexpr size_t SMEM_LIMIT = 224 * 1024;        // most dynamic memory of a plan
// What a launch asks for: with more than eight rows at least so much that no second CTA fits the SM.  Where two fit, those of a launch
// that starts while a quantizer drains pair up on the SMs that come free first and other SMs idle.  us, quantizer and product, two may
// share / one per SM: 9 x 19661 x 4352 34.1 / 23.0, 16 x 35626 x 2816 34.8 / 18.9, 14 x 8993 x 1792 8.4 / 6.7, 12 x 12854 x 768 fp16
// 7.0 / 5.7.  Products back to back without a quantizer overlap less for it: 13 x 6789 x 768 3.2 / 3.5, 14 x 22531 x 768 5.6 / 5.8,
// 9 x 14343 x 3840 12.2 / 12.2.
constexpr size_t OWN_SM = 114 * 1024;
W4A8_PLAN_FN size_t launch_smem(int MH, int S, int nb, int GS, int STAGES) {
    const size_t need = smem_bytes(MH, S, nb, GS, STAGES);
    return MH == 2 && need < OWN_SM ? OWN_SM : need;
}

// Rows up to eight are relayed where a CTA has few tiles (decided in the kernel); for more rows it is another kernel, chosen here.
struct Plan { int MH, GS, STAGES; bool relay; };

// nb groups a row, OUT weight rows, S of 1 to 16 activation rows, `sms` CTAs; max_gs and max_stages (0: as measured) are limits.
// Groups per step: the largest of 16 and 8 that divides the number of groups and fits.  Whether there is a plan does not depend on OUT:
// the ranks of a sharded product come to the same number of launches, whatever their slices.
W4A8_PLAN_FN bool plan_rows(int nb, long OUT, int S, int sms, int max_gs, int max_stages, Plan *p) {
    if (nb <= 0 || nb % 8 != 0) return false;
    const int MH = S > 8 ? 2 : 1;
    // 9 to 16 rows of a matrix with at most two tiles per CTA are relayed, in steps of eight groups.  us, one warp a tile / relay:
    // 16 x 2048 x 8192 16.7 / 11.3, 16 x 4096 x 3840 8.9 / 7.3 (fp16 9.5 / 7.3), 10 x 2500 x 2304 fp16 6.5 / 5.2, 9 x 2048 x 2048
    // 4.7 / 4.2; also where a row has one, three or five steps: 12 x 2254 x 256 2.9 / 2.6, 12 x 405 x 768 3.0 / 2.7, 13 x 1065 x 1280
    // fp16 3.8 / 3.4.  Rows of 16 or 32 groups go in one or two steps of 16 without it (12 x 4000 x 512 2.8 / 3.2).  With three or four
    // tiles two warps each gain nothing (12 x 5120 x 5120 10.6 / 11.0, 16 x 9472 x 4096 9.4 / 10.1).
    const bool narrow = RELAY && MH == 2 && (OUT + 7) / 8 <= (long)sms * 2 * RELAY16_TILES;
    for (int gi = 0; gi < 2; gi++) {
        const int GS = (gi == 0) == (narrow && nb >= 48) ? 8 : 16;
        if (GS > max_gs || nb % GS != 0) continue;
        const int stages[3] = {GS == 16 ? 4 : 8, GS == 16 ? 3 : 6, GS == 16 ? 2 : 3};
        for (int i = 0; i < 3; i++) {
            if (stages[i] > (max_stages > 0 ? max_stages : stages[2])) continue;
            const size_t smem = launch_smem(MH, S, nb, GS, stages[i]);
            if (smem > SMEM_LIMIT) continue;
            p->MH = MH; p->GS = GS; p->STAGES = stages[i];
            // the mailboxes may be what no longer fits (16 rows of 9216): such launches go without
            p->relay = narrow && GS == 8 && i == 2 && smem + static_bytes(MH, true) <= SMEM_CTA;
            return true;
        }
    }
    return false;
}

}  // namespace gemv_mma
}  // namespace w4a8
