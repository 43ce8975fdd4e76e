// Activation quantization, fp32 row -> int8 + per-32-block scale (+ block sums).
// Semantics: reference kernels/quantize_x.cuh:22-39 (d = amax/127.0f, q = rintf(x/d), clamp +-127,
// all-zero block -> q = 0 and d = 0).  HBM-bound: 5.25 bytes moved per element.
#pragma once
#include "common.cuh"

namespace w4a8 {

// Eight threads own one 32-element block: each loads a float4 (16 B), the block maximum and the block
// sum are formed with three xor-shuffles inside the 8-lane group, each thread stores its 4 int8 as one
// 32-bit word.  A warp therefore reads 512 contiguous bytes and writes 128.  UNROLL independent vectors
// per thread are loaded before any is used, to keep enough bytes in flight per SM.  For X aligned to 16 bytes only.  Issue-bound, not HBM-bound, while it
// divided four times per vector; with the reciprocal of quantize4_pack 8192 x 5120 went from 55.2 to 49.0 us (4.0 to
// 4.5 TB/s).
template <int UNROLL>
__global__ void __launch_bounds__(256) quantize_x_q8_vec_kernel(const float4 *__restrict__ X, uint32_t *__restrict__ xq,
                                                                float *__restrict__ xs, int32_t *__restrict__ xsum,
                                                                long nvec /* = S*IN/4, a multiple of 8 */) {
    const long stride = (long)gridDim.x * blockDim.x;
    long i0 = (long)blockIdx.x * blockDim.x + threadIdx.x;
    // Launched while the kernel before it drains; X may come from that kernel and xq may still be read by it.
    pdl_wait();
    // Lets a following kernel that was launched for programmatic dependent launch (the GEMV) become resident and
    // start streaming its weights while this kernel runs; it still waits for this kernel's completion before it
    // reads xq / xs.  Only after the wait above, so that everything issued before this kernel, a weight upload among it,
    // is complete and visible to those early loads.
    pdl_launch_dependents();
    // nvec is a multiple of 8 and i0 - lane is a multiple of 32, so the 8-lane groups are either fully
    // inside or fully outside; shuffles use the full mask with out-of-range lanes carrying zeros.
    for (; i0 - (threadIdx.x & 31) < nvec; i0 += stride * UNROLL) {
        float4 v[UNROLL];
#pragma unroll
        for (int u = 0; u < UNROLL; u++) {
            long i = i0 + u * stride;
            v[u] = (i < nvec) ? __ldcs(X + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < UNROLL; u++) {
            long i = i0 + u * stride;
            float d;
            int sum;
            const uint32_t packed = quantize_block_vec4(v[u], d, sum);
            sum = block_sum(sum);
            if (i < nvec) {
                xq[i] = packed;
                if ((i & 7) == 0) {
                    xs[i >> 3] = d;
                    if (xsum) xsum[i >> 3] = sum;
                }
            }
        }
    }
}

// The same with eight elements a thread, for X aligned to 32 bytes: 56 instead of 96 warp instructions per 128 elements, because four
// lanes share a block's maximum, scale and sum and not eight, maxima take three operands, multiply and fma two elements, and a 256-bit
// load is a whole sector per lane.  What bounds it now is HBM and its latency: 8192 x 5120 44.4 -> 36.3 us in a chain, 5.25 bytes an
// element = 6.1 TB/s of the measured 6.56; 4000 x 3840 18.8 -> 14.2, 2048 x 5120 14.2 -> 9.7, one row of 5120 2.7 -> 2.2.  One vector a
// thread: two, three and four in flight 1 to 5 us more at 8192 rows, and fewer threads hide less in the small cases (16 x 5120 2.9,
// 3.2, 3.7).
constexpr int WIDE_CTAS = 6;                     // of 256 threads on an SM with up to 40 registers (it has 37); a grid of eight per SM is 1.3 waves: 44.0 us
__device__ __forceinline__ void load8(const float *p, float (&v)[8]) {
    asm volatile("ld.global.L1::no_allocate.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "l"(p));
}
__device__ __forceinline__ float max3_abs(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(fabsf(a)), "f"(fabsf(b)), "f"(fabsf(c)));
    return r;
}
__device__ __forceinline__ float max3_abs_nan(float a, float b, float c) {                   // NaN if one of them is
    float r;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(fabsf(a)), "f"(fabsf(b)), "f"(fabsf(c)));
    return r;
}
// quantize4_pack (common.cuh) for eight elements, two at a time.
__device__ __forceinline__ uint2 quantize8_pack(const float (&v)[8], float d, int &sum) {
    constexpr float MAGIC = 12582912.0f, TIE = 0.5f - 0x1p-15f;
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    uint64_t r2, g2;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r2) : "f"(r));
    asm("mov.b64 %0, {%1, %1};" : "=l"(g2) : "f"(MAGIC));
    float m[8], t[8];
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
        uint64_t x2, m2, n2, t2;
        asm("mov.b64 %0, {%1, %2};" : "=l"(x2) : "f"(v[i]), "f"(v[i + 1]));
        asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(m2) : "l"(x2), "l"(r2), "l"(g2));
        asm("mov.b64 {%0, %1}, %2;" : "=f"(m[i]), "=f"(m[i + 1]) : "l"(m2));
        asm("mov.b64 %0, {%1, %2};" : "=l"(n2) : "f"(MAGIC - m[i]), "f"(MAGIC - m[i + 1]));
        asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(t2) : "l"(x2), "l"(r2), "l"(n2));
        asm("mov.b64 {%0, %1}, %2;" : "=f"(t[i]), "=f"(t[i + 1]) : "l"(t2));
    }
    uint2 w;
    w.x = __byte_perm(__byte_perm(__float_as_uint(m[0]), __float_as_uint(m[1]), 0x0040),
                      __byte_perm(__float_as_uint(m[2]), __float_as_uint(m[3]), 0x0040), 0x5410);
    w.y = __byte_perm(__byte_perm(__float_as_uint(m[4]), __float_as_uint(m[5]), 0x0040),
                      __byte_perm(__float_as_uint(m[6]), __float_as_uint(m[7]), 0x0040), 0x5410);
    const float far = max3_abs_nan(max3_abs_nan(t[0], t[1], t[2]), max3_abs_nan(t[3], t[4], t[5]), max3_abs_nan(t[6], t[7], 0.f));
    if (!(far <= TIE && d >= 0x1p-100f && d <= 0x1p100f)) {
        w.x = quantize4_div(make_float4(v[0], v[1], v[2], v[3]), d);
        w.y = quantize4_div(make_float4(v[4], v[5], v[6], v[7]), d);
    }
    sum = __dp4a((int)w.y, 0x01010101, __dp4a((int)w.x, 0x01010101, 0));
    return w;
}
// Eight elements of a 32-element block held by 4 consecutive lanes.  Every lane of the warp calls it; lanes that are not live carry zeros.
__device__ __forceinline__ void quantize_store_vec8(const float (&v)[8], long i, bool live, uint2 *__restrict__ xq, float *__restrict__ xs,
                                                    int32_t *__restrict__ xsum) {
    float amax = max3_abs(max3_abs(v[0], v[1], v[2]), max3_abs(v[3], v[4], v[5]), max3_abs(v[6], v[7], v[7]));     // a block of NaNs keeps its NaN
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    const float d = quant_scale(amax);
    int sum = 0;
    uint2 w = make_uint2(0u, 0u);
    if (amax != 0.0f) w = quantize8_pack(v, d, sum);
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    if (live) {
        xq[i] = w;
        if ((i & 3) == 0) {
            xs[i >> 2] = d;
            if (xsum) xsum[i >> 2] = sum;
        }
    }
}
// Vectors first, first + stride, .. of nvec (a multiple of 4); first - lane is a multiple of 32: the 4-lane groups are inside or outside.
__device__ __forceinline__ void quantize_wide(const float *__restrict__ X, uint2 *__restrict__ xq, float *__restrict__ xs, int32_t *__restrict__ xsum,
                                              long nvec, long first, long stride) {
    for (long i = first; i - (threadIdx.x & 31) < nvec; i += stride) {
        float v[8] = {};
        if (i < nvec) load8(X + i * 8, v);
        quantize_store_vec8(v, i, i < nvec, xq, xs, xsum);
    }
}
__global__ void __launch_bounds__(256, WIDE_CTAS) quantize_x_q8_wide_kernel(const float *__restrict__ X, uint2 *__restrict__ xq, float *__restrict__ xs,
                                                                 int32_t *__restrict__ xsum, long nvec /* = S*IN/8 */) {
    pdl_wait();                  // and what stands at the same place of the kernel above
    pdl_launch_dependents();
    quantize_wide(X, xq, xs, xsum, nvec, (long)blockIdx.x * blockDim.x + threadIdx.x, (long)gridDim.x * blockDim.x);
}

// Same arithmetic with one lane per element (one warp per block), for pointers that are only 4-byte
// aligned: the reference's launcher accepts those.
__global__ void __launch_bounds__(256) quantize_x_q8_scalar_kernel(const float *__restrict__ X, int8_t *__restrict__ xq,
                                                                   float *__restrict__ xs, int32_t *__restrict__ xsum,
                                                                   long nblk) {
    const int lane = threadIdx.x & 31;
    const long wstride = ((long)gridDim.x * blockDim.x) >> 5;
    pdl_wait();
    for (long b = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < nblk; b += wstride) {
        const float x = X[b * QBLK + lane];
        float amax = fabsf(x);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        const float d = amax / 127.0f;
        int q = (amax == 0.0f) ? 0 : (int)rintf(x / d);
        q = max(-127, min(127, q));
        int sum = q;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        xq[b * QBLK + lane] = (int8_t)q;
        if (lane == 0) {
            xs[b] = d;
            if (xsum) xsum[b] = sum;
        }
    }
}

inline int launch_quantize_x(const float *X, int8_t *xq, float *xs, int32_t *xsum, int IN, int S, cudaStream_t st) {
    if (S == 0 || IN == 0) return W4A8_OK;
    const long nblk = (long)S * (IN / QBLK);
    const int sms = sm_count();
    if (aligned(X, 32) && aligned(xq, 8)) {
        const long nvec = nblk * 4, want = (nvec + 255) / 256, cap = (long)sms * WIDE_CTAS;
        cudaError_t e = launch_pdl(quantize_x_q8_wide_kernel, dim3((unsigned)(want < cap ? want : cap)), dim3(256), 0, st, X, reinterpret_cast<uint2 *>(xq), xs, xsum, nvec);
        if (e != cudaSuccess) return cuda_fail(e, "quantize_x_q8 launch");
    } else if (aligned(X, 16) && aligned(xq, 4)) {
        const long nvec = nblk * 8;
        constexpr int U = 4;
        long want = (nvec + 256L * U - 1) / (256L * U);
        long cap = (long)sms * 8;  // 8 CTAs of 256 threads fill an SM
        unsigned grid = (unsigned)(want < cap ? want : cap);
        // programmatic dependent launch: between two GEMVs of a decode step this kernel's own launch latency was exposed
        // (four linears of one row, 5120 x 17408: 68.6 -> 60.1 us; a layer's five matrices at 8 rows: 66.0 -> 59.5 us)
        cudaError_t e = launch_pdl(quantize_x_q8_vec_kernel<U>, dim3(grid), dim3(256), 0, st, reinterpret_cast<const float4 *>(X),
                                   reinterpret_cast<uint32_t *>(xq), xs, xsum, nvec);
        if (e != cudaSuccess) return cuda_fail(e, "quantize_x_q8 launch");
    } else {
        long want = (nblk + 7) / 8;
        long cap = (long)sms * 8;
        unsigned grid = (unsigned)(want < cap ? want : cap);
        cudaError_t e = launch_pdl(quantize_x_q8_scalar_kernel, dim3(grid), dim3(256), 0, st, X, xq, xs, xsum, nblk);
        if (e != cudaSuccess) return cuda_fail(e, "quantize_x_q8 launch");
    }
    return launch_status("quantize_x_q8");
}

}  // namespace w4a8
