// Shared host/device helpers of the W4A8 library (sm_100a only).
#pragma once
#include <cstdint>
#include <cstdio>
#include <cstdarg>
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include "../../include/w4a8_b200.h"

#define W4A8_API extern "C" __attribute__((visibility("default")))

namespace w4a8 {

constexpr int QBLK = W4A8_QBLK;

// ---- host-side error text ----------------------------------------------------------------------
char *err_buf();  // thread-local 512-byte buffer (api.cu)
inline int fail(int code, const char *fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(err_buf(), 512, fmt, ap);
    va_end(ap);
    return code;
}
// The caller learns of e from the return code, so it must not stay behind as the thread's last error, where the next
// call's launch_status would report it for a launch that succeeded.
inline int cuda_fail(cudaError_t e, const char *what) {
    cudaGetLastError();
    return fail(W4A8_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}
// After a kernel launch: reports launch-configuration errors without synchronising.
inline int launch_status(const char *what) {
    cudaError_t e = cudaPeekAtLastError();
    if (e != cudaSuccess) return cuda_fail(e, what);
    return W4A8_OK;
}
inline bool aligned(const void *p, size_t a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; }

// A value per CUDA device, selected by the current device: launch-side caches of per-device facts (function
// attributes such as the dynamic shared-memory opt-in, occupancy answers) must not leak from one GPU to the next in
// a process that drives several.
template <typename T>
struct PerDevice {
    static constexpr int MAX_DEV = 64;
    T v[MAX_DEV] = {};
    T &get() {
        int d = 0;
        if (cudaGetDevice(&d) != cudaSuccess || d < 0 || d >= MAX_DEV) d = 0;
        return v[d];
    }
};

// Number of SMs of the current device (148 on B200), cached per device.
int sm_count();
// W4A8_OK if the current device is compute capability 10.x, else W4A8_ERR_UNSUPPORTED.
int require_sm100();

// ---- programmatic dependent launch ---------------------------------------------------------------
// Kernels that only READ data no earlier kernel of the stream writes (the weights) before they touch anything
// else are launched with the programmatic-stream-serialization attribute: their CTAs may become resident while
// the previous kernel of the stream is still draining, issue their first weight loads, and then block in
// pdl_wait() until that kernel has completed and its writes are visible.  That hides the launch gap and the
// ramp-up of a 10-microsecond kernel behind the tail of its predecessor.  Without the attribute both
// instructions do nothing.  W4A8_PDL=0 in the environment disables the attribute (plain stream order).
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
bool pdl_enabled();   // w4a8_b200.cu

template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, KArgs(args)...);
}

// ---- device-side error word (set when a bounded wait runs out) ---------------------------------
__device__ unsigned int g_dev_error = 0u;  // one translation unit: w4a8_b200.cu includes every kernel file
__device__ __forceinline__ void dev_set_error(unsigned int code) { atomicCAS(&g_dev_error, 0u, code); }

#ifdef __CUDACC__
// ---- weight scale read: float, or __half widened (reference: kernels/qscale.cuh:5-6) -----------
__device__ __forceinline__ float sval(float x) { return x; }
__device__ __forceinline__ float sval(__half x) { return __half2float(x); }

// ---- int4 -> int8 expansion ------------------------------------------------------------------
// One 32-bit word of packed weights holds 8 nibbles: byte j = element 2j (low) and 2j+1 (high).
// Instead of (nibble - 8) the expansion produces 16*(nibble - 8) in each int8 byte: XOR with 8
// turns the nibble into the 4-bit two's-complement code of (nibble - 8), and a nibble sitting in
// the HIGH half of a byte with a zero low half is that value times 16.  Integer dot products are
// then 16x the true ones (still exact: |16*D| <= 520,192) and the factor 1/16 is folded into the
// fp32 scale, where it is exact.  Cost: 3 logic ops per 8 weights, no per-byte subtraction.
//   even: bytes = 16*w[0], 16*w[2], 16*w[4], 16*w[6]   (the word's low nibbles)
//   odd : bytes = 16*w[1], 16*w[3], 16*w[5], 16*w[7]   (the word's high nibbles)
// The three-input logic instruction by hand: from the C expression the compiler makes two instructions of one constant each, ten for
// the two words of a tensor instruction's operand instead of six (counted under ncu).  Half-rate ones: they are what the decode
// kernels for 8 and 16 rows and the experts' run out of.  us, expression / this: 16 x 17408 x 5120 fp16 scales three times 65.8 / 58.9,
// expert block of 8 rows 40.6 / 38.6, 333 x 15360 x 3840 122.9 / 118.9, one row x 151936 x 5120 71.1 / 69.6.
__device__ __forceinline__ uint32_t and_xor(uint32_t a, uint32_t mask, uint32_t x) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0x6a;" : "=r"(r) : "r"(a), "r"(mask), "r"(x));
    return r;
}
__device__ __forceinline__ void unpack8_x16(uint32_t w, uint32_t &even, uint32_t &odd) {
    odd = and_xor(w, 0xF0F0F0F0u, 0x80808080u);
    even = and_xor(w << 4, 0xF0F0F0F0u, 0x80808080u);
}
// The same, left to the compiler.
__device__ __forceinline__ void unpack8_x16_expr(uint32_t w, uint32_t &even, uint32_t &odd) {
    odd = (w & 0xF0F0F0F0u) ^ 0x80808080u;
    even = ((w << 4) & 0xF0F0F0F0u) ^ 0x80808080u;
}
// The same 8 weights in element order (for tensor-core operands): lo = 16*w[0..3], hi = 16*w[4..7].
__device__ __forceinline__ void unpack8_x16_seq(uint32_t w, uint32_t &lo, uint32_t &hi) {
    uint32_t even, odd;
    unpack8_x16(w, even, odd);
    lo = __byte_perm(even, odd, 0x5140);  // e0 o0 e1 o1
    hi = __byte_perm(even, odd, 0x7362);  // e2 o2 e3 o3
}
// d = amax / 127, the IEEE quotient.  Inside [2^-100, 2^100] by one Markstein correction step (quotient estimate times the
// rounded reciprocal, exact remainder by fma, second fma): three instructions, and equal to the division for every
// mantissa (checked over all 2^23 of them; scaling by powers of two changes nothing while no result is subnormal).
__device__ __forceinline__ float quant_scale(float amax) {
    if (amax >= 0x1p-100f && amax <= 0x1p100f) {
        constexpr float c = 1.0f / 127.0f;
        const float q = amax * c;
        return fmaf(fmaf(-127.0f, q, amax), c, q);
    }
    return amax / 127.0f;
}
// Four quantized activations of one float4: q = rintf(x / d) clamped to +-127 (kernels/quantize_x.cuh:36-37), packed into
// one word (byte i = q_i).  cvt.rni.sat.s8.f32 rounds to nearest even, converts and saturates (a NaN quotient — amax
// infinite, or 0 / 0 — gives 0 either way); the saturation stops at -128 and the definition at -127.  While d is a normal
// number the quotient is at most 127 * (1 + 2^-23) in magnitude, because |x| <= amax and d = amax / 127 rounded; a subnormal
// d is rounded so coarsely that it reaches 190, so the lower bound is taken here, on the path that all such d take.
__device__ __forceinline__ int quantize1_div(float x, float d) {
    int q;
    asm("cvt.rni.sat.s8.f32 %0, %1;" : "=r"(q) : "f"(x / d));
    return max(q, -127);
}
__device__ __noinline__ uint32_t quantize4_div(float4 v, float d) {
    const int q0 = quantize1_div(v.x, d), q1 = quantize1_div(v.y, d), q2 = quantize1_div(v.z, d), q3 = quantize1_div(v.w, d);
    const uint32_t lo = __byte_perm((uint32_t)q0, (uint32_t)q1, 0x0040), hi = __byte_perm((uint32_t)q2, (uint32_t)q3, 0x0040);
    return __byte_perm(lo, hi, 0x5410);
}
// The same without the four divisions, which made the quantizer issue-bound (117 warp instructions per 128 elements): with
// r = 1/d to one ulp (rcp.approx: relative error at most 2^-23), m = fma(x, r, 1.5 * 2^23) holds the integer nearest to x*r
// in its low byte, and t = x*r - q is its distance.  |x*r - x/d| <= 127 * 2^-23 = 1.6e-5 and the fp32 quotient is within
// 2^-18 = 3.8e-6 of x/d, so where |t| <= 0.5 - 2^-15 no half-integer lies between x*r and the fp32 quotient and both
// round to the same q, at most 127 in magnitude.  The other elements (about 6 in 10^5), d outside the range in which r keeps
// its accuracy, and anything that is not finite take the divisions.
__device__ __forceinline__ uint32_t quantize4_pack(float4 v, float d, int &sum) {
    constexpr float MAGIC = 12582912.0f, TIE = 0.5f - 0x1p-15f;
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    const float m0 = fmaf(v.x, r, MAGIC), m1 = fmaf(v.y, r, MAGIC), m2 = fmaf(v.z, r, MAGIC), m3 = fmaf(v.w, r, MAGIC);
    const float t0 = fmaf(v.x, r, MAGIC - m0), t1 = fmaf(v.y, r, MAGIC - m1), t2 = fmaf(v.z, r, MAGIC - m2), t3 = fmaf(v.w, r, MAGIC - m3);
    uint32_t w = __byte_perm(__byte_perm(__float_as_uint(m0), __float_as_uint(m1), 0x0040),
                             __byte_perm(__float_as_uint(m2), __float_as_uint(m3), 0x0040), 0x5410);
    const bool sure = fabsf(t0) <= TIE && fabsf(t1) <= TIE && fabsf(t2) <= TIE && fabsf(t3) <= TIE && d >= 0x1p-100f && d <= 0x1p100f;
    if (!sure) w = quantize4_div(v, d);
    sum = __dp4a((int)w, 0x01010101, 0);
    return w;
}
// Four elements of a 32-element block held by 8 consecutive lanes (d = amax / 127, q = rintf(x / d) clamped, zero block -> zeros):
// the packed word, the block's scale and the sum of these four.  Every lane of the warp calls it.
__device__ __forceinline__ uint32_t quantize_block_vec4(float4 v, float &d, int &sum) {
    float amax = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
    d = quant_scale(amax);
    sum = 0;
    return amax != 0.0f ? quantize4_pack(v, d, sum) : 0u;
}
// The block's sum from the 8 lanes' sums.
__device__ __forceinline__ int block_sum(int sum) {
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    return sum + __shfl_xor_sync(0xffffffffu, sum, 4);
}
// Activation bytes x[0..7] (two words) split the same way: even = x0 x2 x4 x6, odd = x1 x3 x5 x7.
__device__ __forceinline__ void split_even_odd(uint32_t x0, uint32_t x1, uint32_t &even, uint32_t &odd) {
    even = __byte_perm(x0, x1, 0x6420);
    odd = __byte_perm(x0, x1, 0x7531);
}
#endif

}  // namespace w4a8
