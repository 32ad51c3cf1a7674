// common.cuh -- shared device helpers of libgsea103 (GB300 / sm_103a).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace gsea {

constexpr uint32_t kFullMask = 0xffffffffu;

// ---------------------------------------------------------------------------
// Exact IEEE operations.  The reference's metric arithmetic is reproduced
// bit for bit, so no product may be fused into an addition: the *_rn
// intrinsics are never contracted into FMA by the compiler.
template <class T> struct Exact;
template <> struct Exact<float> {
    static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
    static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
    static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
    static __device__ __forceinline__ float div(float a, float b) { return __fdiv_rn(a, b); }
    static __device__ __forceinline__ float sqrt(float a) { return __fsqrt_rn(a); }
    // floor of a standard deviation / variance: (T)(c * |m|) evaluated in double
    // (functors.cuh:46-47, 72-73 multiply a double literal by a float)
    // In fp32: the product with the constant in two parts, whose sum is off
    // the exact product by less than 2^-45 of it; wherever that could decide
    // the rounding (or the value is outside the plain range) the double
    // product itself is taken.  Its three FP64-pipe operations on every key
    // took 0.24 ms of that pipe per 20,000 x 1,000 keys.
    static __device__ __forceinline__ float low(double c, float m) {
        const float ch = (float)c, cl = (float)(c - (double)ch);  // constants
        const float hi = __fmul_rn(m, ch);
        const float t = __fmaf_rn(m, cl, __fmaf_rn(m, ch, -hi));
        const float r = __fadd_rn(hi, t);
        const float rem = fabsf(__fadd_rn(__fsub_rn(hi, r), t));  // what the rounding to r left
        const uint32_t ex = __float_as_uint(r) & 0x7f800000u;
        const float half = __uint_as_float(ex - (24u << 23));     // half a unit in the last place of r
        // also taken next to a power of two, where the unit changes
        if (ex < (60u << 23) || ex > (200u << 23) || (__float_as_uint(r) & 0x007fffffu) == 0u ||
            fabsf(__fsub_rn(rem, half)) < __fmul_rn(half, 1.52587890625e-5f))
            return low_double(c, m);
        return r;
    }
    // out of line: inlined, the compiler runs it every time and selects
    static __device__ __noinline__ float low_double(double c, float m) {
        return __double2float_rn(__dmul_rn(c, (double)m));
    }
    // culog(q) * 1.44269504089 : float log, double product, rounded to float
    // (functors.cuh:24-29, math_helpers.cuh:5, 37-40)
    static __device__ __forceinline__ float log2q(float q) {
        return __double2float_rn(__dmul_rn((double)logf(q), 1.44269504089));
    }
};
template <> struct Exact<double> {
    static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
    static __device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
    static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
    static __device__ __forceinline__ double div(double a, double b) { return __ddiv_rn(a, b); }
    static __device__ __forceinline__ double sqrt(double a) { return __dsqrt_rn(a); }
    static __device__ __forceinline__ double low(double c, double m) { return __dmul_rn(c, m); }
    static __device__ __forceinline__ double log2q(double q) { return __dmul_rn(log(q), 1.44269504089); }
};

// cuabs of math_helpers.cuh:10-13 (keeps -0.0 and NaN as they are)
template <class T> __device__ __forceinline__ T cuabs(T x) { return x < T(0) ? -x : x; }

// ---------------------------------------------------------------------------
// Radix order of IEEE keys: unsigned ascending order of radix_bits(x) equals
// ascending value order with -0 < +0 and NaNs at the two ends, which is the
// order CUB's radix sort gives the reference GPU path (batched_sort.cuh:144).
// The bits are taken by a move the compiler does not look through: where the
// value is used as a number too, it rewrites "sign bit set" as a negated
// absolute value in floating point, which gives a NaN another sign (seen with
// doubles: the key of a NaN differed from that of an equal NaN).
__device__ __forceinline__ uint32_t bits_of(float f) {
    uint32_t u;
    asm("mov.b32 %0, %1;" : "=r"(u) : "f"(f));
    return u;
}
__device__ __forceinline__ unsigned long long bits_of(double f) {
    unsigned long long u;
    asm("mov.b64 %0, %1;" : "=l"(u) : "d"(f));
    return u;
}
template <class T> struct RadixKey;
template <> struct RadixKey<float> {
    using U = uint32_t;
    static __device__ __forceinline__ U from(float f, bool descending) {
        U u = bits_of(f);
        u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
        return descending ? ~u : u;
    }
};
template <> struct RadixKey<double> {
    using U = unsigned long long;
    static __device__ __forceinline__ U from(double f, bool descending) {
        U u = bits_of(f);
        u = (u & 0x8000000000000000ull) ? ~u : (u | 0x8000000000000000ull);
        return descending ? ~u : u;
    }
};

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm volatile("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

}  // namespace gsea
