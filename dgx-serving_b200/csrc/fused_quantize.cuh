// Producer + quantize_x fusions: RMSNorm -> quantize and SwiGLU / GeGLU -> quantize in one kernel each.
// The reference's graphs always run norm -> quantize_x -> matmul and activation -> quantize_x -> down projection
// (models/qwen35_decode.cu:148-149, 215-218) as separate kernels with an fp32 round trip between them.  The fused
// kernels repeat the unfused element math exactly — the row sum of squares in the order of the reference's
// rmsnorm_kernel (kernels/rmsnorm.cuh:8-20: 256 threads, thread t adds elements t, t+256, ... then
// block_reduce_sum of kernels/reduce.cuh:11-24), the same rsqrtf / expf / tanhf calls and the same products — so
// xq, xs, xsum (and the optional fp32 copy of the intermediate) equal the two-kernel sequence bit for bit.
#pragma once
#include "common.cuh"
#include "quantize_x.cuh"

namespace w4a8 {

// One float4 of a 32-element block held by 8 consecutive lanes, outputs as in quantize_x_q8_vec_kernel.  Every lane of the
// warp must call it; lanes with live == false carry zeros and store nothing.
__device__ __forceinline__ void quantize_store_vec4(float4 v, long i, bool live, uint32_t *__restrict__ xq,
                                                    float *__restrict__ xs, int32_t *__restrict__ xsum) {
    float d;
    int sum;
    const uint32_t packed = quantize_block_vec4(v, d, sum);
    sum = block_sum(sum);
    if (live) {
        xq[i] = packed;
        if ((i & 7) == 0) {
            xs[i >> 3] = d;
            if (xsum) xsum[i >> 3] = sum;
        }
    }
}

// The same for a row that stays in shared memory (the prologue of a GEMV that quantizes its own activation row): word i
// of the row -> xrow[i], the scale of block i / 8 -> xs_row[i / 8]; g_xq / g_xs (null: skipped) receive the same values.
__device__ __forceinline__ void quantize_row_vec4(float4 v, int i, bool live, uint32_t *xrow, float *xs_row,
                                                  uint32_t *__restrict__ g_xq, float *__restrict__ g_xs) {
    float d;
    int sum;
    const uint32_t packed = quantize_block_vec4(v, d, sum);
    if (live) {
        xrow[i] = packed;
        if (g_xq) g_xq[i] = packed;
        if ((i & 7) == 0) {
            xs_row[i >> 3] = d;
            if (g_xs) g_xs[i >> 3] = d;
        }
    }
}

// An fp32 row that a GEMV quantizes itself instead of waiting for a launch of quantize_x: every CTA quantizes the whole row for
// its own shared memory, the first one also stores xq / xs / xsum (null: skipped) for the caller.
struct RowSrc {
    const float *x = nullptr;
    uint32_t *xq = nullptr;
    float *xs = nullptr;
    int32_t *xsum = nullptr;
};
// The float4s i = tid, tid + NT, ... of the row.  load() asks for the first UB of them (ahead of the weights, so that they do not
// queue behind them); quantize() calls put(i, word, d, live) with four quantized elements and the scale of their block.  Every lane
// of a warp reaches put together, live == false past the end.  nvec = row length / 4, a multiple of 8.
template <int NT, int UB>
struct RowQuantizer {
    float4 v[UB];
    __device__ __forceinline__ void load(const RowSrc &src, int nvec, int i0) {
        const float4 *x4 = reinterpret_cast<const float4 *>(src.x);
#pragma unroll
        for (int u = 0; u < UB; u++) v[u] = i0 + u * NT < nvec ? x4[i0 + u * NT] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    template <class F>
    __device__ __forceinline__ void quantize(const RowSrc &src, int nvec, int tid, bool store, F &&put) {
        const int lane = tid & 31;
        for (int i0 = tid; i0 - lane < nvec; i0 += NT * UB) {
            if (i0 != tid) load(src, nvec, i0);
#pragma unroll
            for (int u = 0; u < UB; u++) {
                const int i = i0 + u * NT;
                if (i - lane < nvec) {                                              // the same for the whole warp
                    const bool live = i < nvec;
                    float d;
                    int sum;
                    const uint32_t packed = quantize_block_vec4(v[u], d, sum);
                    put(i, packed, d, live);
                    if (store) {
                        sum = block_sum(sum);
                        if (live) {
                            src.xq[i] = packed;
                            if ((i & 7) == 0) {
                                src.xs[i >> 3] = d;
                                if (src.xsum) src.xsum[i >> 3] = sum;
                            }
                        }
                    }
                }
            }
        }
    }
};

// VARIANT 0: y = x * inv * W (launch_rmsnorm); 1: y = x * inv * (1 + W) (launch_rmsnorm_zc); 2: y = x * inv
// (launch_rmsnorm_noscale).  One CTA of 256 threads per row, as in the reference (the reduction order depends on it).
// Bound by latency: a decode step has a few rows, each on one SM, and every dependent trip to L2 costs about 0.4 us.  So DEEP has
// all loads of a trip of both passes in flight at once: UB strided elements for the sum, and UV float4 of x and W, the latter
// asked for before the sum is reduced (W does not depend on it).  An MLP block of one row, 5120 x 17408: 47.0 -> 43.8 us; 64 rows
// of 17408 11.0 -> 9.2.  With more rows it is CTAs that hide the latency, and the registers of deep batches cost more CTAs than
// they give: see launch_rmsnorm_quantize for the line.
template <int VARIANT, bool DEEP>
__global__ void __launch_bounds__(256) rmsnorm_quantize_kernel(const float *__restrict__ X, const float *__restrict__ W, float eps,
                                                               float *__restrict__ Y, uint32_t *__restrict__ xq, float *__restrict__ xs,
                                                               int32_t *__restrict__ xsum, int hh) {
    __shared__ float sh[32];
    __shared__ float inv_s;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const size_t row = blockIdx.x;
    const float *xr = X + row * hh;
    pdl_wait();              // X may come from the kernel before this one; see quantize_x_q8_vec_kernel for the order
    pdl_launch_dependents();
    const int n4 = hh >> 2;                      // a multiple of 8: every 8-lane group is one whole block
    const float4 *x4 = reinterpret_cast<const float4 *>(xr);
    const float4 *w4 = reinterpret_cast<const float4 *>(W);
    constexpr int UB = 32, UV = DEEP ? 8 : 1;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 xv[UV], wv[UV];
    auto fetch = [&](int j) {
#pragma unroll
        for (int u = 0; u < UV; u++) {
            xv[u] = wv[u] = zero;
            if (j + u * 256 < n4) {
                xv[u] = x4[j + u * 256];
                if (VARIANT != 2) wv[u] = w4[j + u * 256];
            }
        }
    };
    float ss = 0.f;
    if constexpr (DEEP) {
        for (int i0 = tid; i0 < hh; i0 += 256 * UB) {
            float v[UB];
#pragma unroll
            for (int u = 0; u < UB; u++) v[u] = i0 + u * 256 < hh ? xr[i0 + u * 256] : 0.f;
            if (i0 == tid) fetch(tid);
#pragma unroll
            for (int u = 0; u < UB; u++) ss = i0 + u * 256 < hh ? fmaf(v[u], v[u], ss) : ss;
        }
    } else {
        for (int i = tid; i < hh; i += 256) { const float v = xr[i]; ss = fmaf(v, v, ss); }
    }
    // block_reduce_sum of the reference: shfl_down tree per warp, partials through shared memory, warp 0 adds them
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_down_sync(0xffffffffu, ss, o);
    if (lane == 0) sh[wid] = ss;
    __syncthreads();
    ss = (tid < 8) ? sh[lane] : 0.0f;
    if (wid == 0) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_down_sync(0xffffffffu, ss, o);
        if (lane == 0) inv_s = rsqrtf(ss / hh + eps);
    }
    __syncthreads();
    const float inv = inv_s;
    for (int j0 = tid; j0 - lane < n4; j0 += 256 * UV) {
        if (!DEEP || j0 != tid) fetch(j0);
#pragma unroll
        for (int u = 0; u < UV; u++) {
            const int j = j0 + u * 256;
            if (j - lane < n4) {                 // the same for the whole warp
                const bool live = j < n4;
                const float4 x = xv[u], w = wv[u];
                float4 y = zero;
                if (live) {
                    if (VARIANT == 2) y = make_float4(x.x * inv, x.y * inv, x.z * inv, x.w * inv);
                    else if (VARIANT == 0) y = make_float4(x.x * inv * w.x, x.y * inv * w.y, x.z * inv * w.z, x.w * inv * w.w);
                    else y = make_float4(x.x * inv * (1.0f + w.x), x.y * inv * (1.0f + w.y), x.z * inv * (1.0f + w.z), x.w * inv * (1.0f + w.w));
                    if (Y) reinterpret_cast<float4 *>(Y + row * hh)[j] = y;
                }
                quantize_store_vec4(y, (long)(row * n4) + j, live, xq, xs, xsum);
            }
        }
    }
}

// ACT 0: y = silu(g) * u (kernels/swiglu.cuh:5-8); 1: y = gelu_tanh(g) * u (kernels/swiglu.cuh:19-27).
template <int ACT>
__device__ __forceinline__ float glu_value(float g, float u) {
    if (ACT == 0) { const float s = g / (1.0f + expf(-g)); return s * u; }
    const float t = tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g));
    return 0.5f * g * (1.0f + t) * u;
}
template <int ACT>
__global__ void __launch_bounds__(256) glu_quantize_kernel(const float4 *__restrict__ G, const float4 *__restrict__ U, float4 *__restrict__ Y,
                                                           uint32_t *__restrict__ xq, float *__restrict__ xs, int32_t *__restrict__ xsum,
                                                           long nvec /* = S*IN/4, a multiple of 8 */, int row_vecs, long pitch_vecs) {
    // row_vecs = IN/4; rows of G and U start pitch_vecs float4s apart (== row_vecs: dense; a fused gate|up tensor
    // [S][2*IN] has pitch 2*IN/4 and U = G + IN)
    const long stride = (long)gridDim.x * blockDim.x;
    pdl_wait();   // G and U come from the kernel before this one
    pdl_launch_dependents();
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i - (threadIdx.x & 31) < nvec; i += stride) {
        const bool live = i < nvec;
        float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
        if (live) {
            const long src = pitch_vecs == row_vecs ? i : (i / row_vecs) * pitch_vecs + (i % row_vecs);
            const float4 g = G[src], u = U[src];
            y = make_float4(glu_value<ACT>(g.x, u.x), glu_value<ACT>(g.y, u.y), glu_value<ACT>(g.z, u.z), glu_value<ACT>(g.w, u.w));
            if (Y) Y[i] = y;
        }
        quantize_store_vec4(y, i, live, xq, xs, xsum);
    }
}

// The same with eight elements a thread (quantize_x_q8_wide_kernel): G, U and the pitch aligned to 32 bytes.  Rows by 32-bit division: the
// 64-bit one of the kernel above is a call of a hundred instructions.  4096 rows of 768, pitch 1536: 10.8 us, 8.4 so (ncu, from DRAM).
template <int ACT>
__global__ void __launch_bounds__(256) glu_quantize_wide_kernel(const float *__restrict__ G, const float *__restrict__ U, float *__restrict__ Y,
                                                                uint2 *__restrict__ xq, float *__restrict__ xs, int32_t *__restrict__ xsum,
                                                                uint32_t nvec /* = S*IN/8 < 2^31, a multiple of 4 */, uint32_t row_vecs, uint32_t pitch_vecs) {
    const uint32_t stride = gridDim.x * blockDim.x;
    pdl_wait();   // G and U come from the kernel before this one
    pdl_launch_dependents();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i - (threadIdx.x & 31) < nvec; i += stride) {
        const bool live = i < nvec;
        float y[8] = {};
        if (live) {
            const size_t src = pitch_vecs == row_vecs ? i : (size_t)(i / row_vecs) * pitch_vecs + i % row_vecs;
            float g[8], u[8];
            load8(G + src * 8, g);
            load8(U + src * 8, u);
#pragma unroll
            for (int k = 0; k < 8; k++) y[k] = glu_value<ACT>(g[k], u[k]);
            if (Y) {
                *reinterpret_cast<float4 *>(Y + (size_t)i * 8) = make_float4(y[0], y[1], y[2], y[3]);
                *reinterpret_cast<float4 *>(Y + (size_t)i * 8 + 4) = make_float4(y[4], y[5], y[6], y[7]);
            }
        }
        quantize_store_vec8(y, i, live, xq, xs, xsum);
    }
}

inline int launch_rmsnorm_quantize(const float *X, const float *W, float eps, int variant, float *Y, int8_t *xq, float *xs,
                                   int32_t *xsum, int IN, int S, cudaStream_t st) {
    uint32_t *q = reinterpret_cast<uint32_t *>(xq);
    // DEEP while its CTAs (151 registers a thread, 128 without a weight vector: one and two per SM) are one wave and the row is
    // longer than the four elements a thread that the plain loop has in flight anyway.  us, DEEP / plain, rows x length: 1 x 1024
    // 1.85 / 1.65, 1 x 1280 2.07 / 2.26, 148 x 5120 3.5 / 4.3, 149 x 5120 5.8 / 4.3, 296 x 17408 17.0 / 11.3, 400 x 5120 9.1 / 4.8;
    // no weights: 296 x 2048 2.84 / 2.67, 296 x 3008 3.32 / 3.69, 296 x 5120 4.0 / 4.4, 297 x 5120 6.1 / 4.4.
    const int sms = sm_count();
    const bool deep = S <= sms ? IN > 1024 : variant == 2 && S <= 2 * sms && IN > 2048;
    auto kern = variant == 0 ? rmsnorm_quantize_kernel<0, false> : variant == 1 ? rmsnorm_quantize_kernel<1, false> : rmsnorm_quantize_kernel<2, false>;
    if (deep) kern = variant == 0 ? rmsnorm_quantize_kernel<0, true> : variant == 1 ? rmsnorm_quantize_kernel<1, true> : rmsnorm_quantize_kernel<2, true>;
    cudaError_t e = launch_pdl(kern, dim3((unsigned)S), dim3(256), 0, st, X, W, eps, Y, q, xs, xsum, IN);
    if (e != cudaSuccess) return cuda_fail(e, "rmsnorm_quantize_x_q8 launch");
    return launch_status("rmsnorm_quantize_x_q8");
}

// Eight elements a thread or four: `ctas` CTAs of the wide kernel, each with the work of two narrow ones.  With few of them per SM what
// counts is how evenly they divide over the SMs, and wide ones divide worse.  us, narrow / wide, SwiGLU, by wide CTAs: 170 1.91 / 2.31, 211 2.05 / 2.43, 261 2.64 / 2.41, 401 2.70 / 2.77, 552 3.38 / 3.14, 723 3.89 / 4.25, 869 4.55 / 4.40,
// 938 4.64 / 4.44, 1255 5.99 / 4.78, 4236 18.6 / 12.7.  GeGLU, whose tanh costs more than the loads: 180 1.97 / 2.15, 203 1.95 / 2.20,
// 224 2.60 / 2.29, 356 2.73 / 2.62, 651 3.83 / 4.21, 810 4.33 / 4.18, 4153 18.5 / 12.5.
constexpr bool glu_takes_wide(long ctas, int sms, int act) {
    const long per_sm = (ctas + sms - 1) / sms;
    if (act == 1) return 2 * ctas > 3L * sms && per_sm != 5;
    return per_sm > 6 || (per_sm % 2 == 0 && 2 * ctas > (2 * per_sm - 1) * sms);
}

inline int launch_glu_quantize(const float *G, const float *U, int act, float *Y, int8_t *xq, float *xs, int32_t *xsum, int IN,
                               int S, cudaStream_t st, long pitch = 0 /* floats between rows of G / U; 0 = IN */) {
    const long n8 = (long)S * IN / 8, w8 = (n8 + 255) / 256, c8 = (long)sm_count() * 8;
    if (glu_takes_wide(w8, sm_count(), act) && aligned(G, 32) && aligned(U, 32) && aligned(xq, 8) && pitch % 8 == 0 && (long)S * IN < (1L << 33)) {
        const cudaError_t e = launch_pdl(act == 0 ? glu_quantize_wide_kernel<0> : glu_quantize_wide_kernel<1>, dim3((unsigned)(w8 < c8 ? w8 : c8)), dim3(256), 0, st,
                                         G, U, Y, reinterpret_cast<uint2 *>(xq), xs, xsum, (uint32_t)n8, (uint32_t)(IN / 8), (uint32_t)((pitch > 0 ? pitch : IN) / 8));
        if (e != cudaSuccess) return cuda_fail(e, "glu_quantize_x_q8 launch");
        return launch_status("glu_quantize_x_q8");
    }
    const long nvec = (long)S * IN / 4;
    long want = (nvec + 255) / 256, cap = (long)sm_count() * 8;
    const unsigned grid = (unsigned)(want < cap ? want : cap);
    const float4 *g = reinterpret_cast<const float4 *>(G), *u = reinterpret_cast<const float4 *>(U);
    float4 *y = reinterpret_cast<float4 *>(Y);
    uint32_t *q = reinterpret_cast<uint32_t *>(xq);
    const long pv = (pitch > 0 ? pitch : IN) / 4;
    cudaError_t e = launch_pdl(act == 0 ? glu_quantize_kernel<0> : glu_quantize_kernel<1>, dim3(grid), dim3(256), 0, st, g, u, y, q, xs, xsum, nvec, IN / 4, pv);
    if (e != cudaSuccess) return cuda_fail(e, "glu_quantize_x_q8 launch");
    return launch_status("glu_quantize_x_q8");
}

}  // namespace w4a8
