// k_metric.cuh -- plain-form class statistics and ranking metric.
//
// For every (permutation, gene) the kernel accumulates class-A / class-B
// statistics over the samples in index order and finalises one of the 14
// reference metrics, reproducing the reference arithmetic operation by
// operation (src/include/functors.cuh:10-433, dispatch
// src/include/correlate_genes.cuh:166-295):
//
//   accumulators  naive (87-124)   kahan (126-176)  onepass (178-229)
//                 twopass (232-295) overkill (297-375) knuth (377-433)
//   combiners     difference (10-15) quotient (17-22) log2 quotient (24-29)
//                 signal2noise, fixlow (31-54)  T test, fixlow (57-80)
//
// All statistics are biased (the reference never forwards `biased`, so the
// accumulators use their default biased=true).  Every product is rounded
// before it is added (Exact<T>), matching the reference's CPU arithmetic.
//
// Work decomposition (GB300).  The class of a sample is the same for every
// gene, so a warp owns a few permutations and its lanes the genes: the class
// bits of the samples select one of sixteen code paths (one indirect branch,
// never divergent), and a path updates each permutation's statistics of the
// sample's own class and nothing else -- no selects, no arithmetic with 0/1
// weights on the other class.  That halves the FP32 work of the selecting
// form for the two-pass metrics (4 operations per gene, sample and
// permutation instead of 8); the FP64 work is the operations themselves.
// fp32 lanes hold their genes as pairs, updated by the paired FP32
// instructions.  The warps of a block share a tile of the expression table,
// copied to shared memory 32 samples at a time (cp.async, two buffers), so
// the table is read from L2 once per block of 16 (fp32) or 32 permutations
// and pass.
#pragma once
#include <algorithm>
#include <type_traits>

#include "bulk.cuh"
#include "common.cuh"
#include "kernels.h"

namespace gsea {

enum AccKind { ACC_NAIVE, ACC_KAHAN, ACC_ONEPASS, ACC_TWOPASS, ACC_KNUTH, ACC_OVERKILL };
enum CombKind { COMB_DIFF, COMB_RATIO, COMB_LOG2, COMB_S2N, COMB_TTEST };

// Division by a class size: the correctly rounded quotient from the rounded
// reciprocal and one exact remainder (Markstein's method; a quotient by an
// integer below 2^13 is never close enough to a rounding boundary for the
// remainder's correction to decide it wrongly).  Values whose remainder could
// leave the normal range are divided by the general operation.
template <class T>
struct ClassSize {
    T n;
    __device__ __forceinline__ explicit ClassSize(T v) : n(v) {}
    __device__ __forceinline__ T divides(T x) const { return Exact<T>::div(x, n); }
};
template <>
struct ClassSize<float> {
    float n, r;
    __device__ __forceinline__ explicit ClassSize(float v) {
        n = v;
        r = __frcp_rn(v);
    }
    __device__ __forceinline__ float divides(float x) const {
        const float q = __fmul_rn(x, r);
        const float f = __fmaf_rn(__fmaf_rn(-q, n, x), r, q);
        const float ax = fabsf(x);
        if ((ax > 1e-25f && ax < 1e30f) || __float_as_uint(x) == 0u) return f;
        return general(x, n);
    }
    static __device__ __noinline__ float general(float x, float n) { return __fdiv_rn(x, n); }
};

template <class T>
__device__ __forceinline__ T combine(int comb, T mA, T vA, const ClassSize<T>& nA, T mB, T vB,
                                     const ClassSize<T>& nB) {
    using E = Exact<T>;
    if (comb == COMB_DIFF) return E::sub(mA, mB);
    if (comb == COMB_RATIO) return E::div(mA, mB);
    if (comb == COMB_LOG2) return E::log2q(E::div(mA, mB));
    if (comb == COMB_S2N) {
        T sA = E::sqrt(vA), sB = E::sqrt(vB);
        const T lowA = E::low(0.2, cuabs(mA));
        const T lowB = E::low(0.2, cuabs(mB));
        sA = lowA < sA ? sA : lowA;
        sB = lowB < sB ? sB : lowB;
        return E::div(E::sub(mA, mB), E::add(sA, sB));
    }
    // COMB_TTEST
    T wA = vA, wB = vB;
    const T lowA = E::low(0.04, cuabs(mA));
    const T lowB = E::low(0.04, cuabs(mB));
    wA = lowA < wA ? wA : lowA;
    wB = lowB < wB ? wB : lowB;
    return E::div(E::sub(mA, mB), E::sqrt(E::add(nA.divides(wA), nB.divides(wB))));
}

// NaN keys (0/0 in the ratio metrics, log of a negative mean, ...) are
// written as the positive all-ones NaN, whatever payload the arithmetic gave:
// the radix order then ranks every NaN first (descending) in gene order, the
// order CUDA's canonical NaN gets from the reference's GPU sort, on any host.
__device__ __forceinline__ float canonical_nan(float v) { return v != v ? __uint_as_float(0x7fffffffu) : v; }
__device__ __forceinline__ double canonical_nan(double v) {
    return v != v ? __longlong_as_double(0x7fffffffffffffffll) : v;
}

// A lane's genes as vectors: pairs of floats (paired FP32 instructions, each
// half rounded on its own), single doubles.
template <class T> struct Vec;
template <> struct Vec<float> {
    using V = unsigned long long;
    static constexpr int kLanes = 2;
    static __device__ __forceinline__ V zero() { return 0ull; }
    static __device__ __forceinline__ V pack(const float* f) {
        V r;
        asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(f[0]), "f"(f[1]));
        return r;
    }
    static __device__ __forceinline__ void unpack(V v, float* f) {
        asm("mov.b64 {%0, %1}, %2;" : "=f"(f[0]), "=f"(f[1]) : "l"(v));
    }
    static __device__ __forceinline__ V add(V a, V b) {
        V d;
        asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
        return d;
    }
    static __device__ __forceinline__ V sub(V a, V b) {
        V d;
        asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
        return d;
    }
    static __device__ __forceinline__ V mul(V a, V b) {
        V d;
        asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
        return d;
    }
    // acc + prod for a product of mul(): the assembler fuses a paired multiply
    // and add into one rounding (it does not for the scalar instructions), but
    // not a multiply into a multiply-add by a `one` it does not know
    static __device__ __forceinline__ V add_product(V acc, V prod, V one) {
        V d;
        asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(one), "l"(prod), "l"(acc));
        return d;
    }
    static __device__ __forceinline__ V runtime_one() {
        const float f[2] = {(float)blockDim.z, (float)blockDim.z};  // 1
        return pack(f);
    }
};
template <> struct Vec<double> {
    using V = double;
    static constexpr int kLanes = 1;
    static __device__ __forceinline__ V zero() { return 0.0; }
    static __device__ __forceinline__ V pack(const double* f) { return f[0]; }
    static __device__ __forceinline__ void unpack(V v, double* f) { f[0] = v; }
    static __device__ __forceinline__ V add(V a, V b) { return __dadd_rn(a, b); }
    static __device__ __forceinline__ V sub(V a, V b) { return __dsub_rn(a, b); }
    static __device__ __forceinline__ V mul(V a, V b) { return __dmul_rn(a, b); }
    static __device__ __forceinline__ V add_product(V acc, V prod, V) { return __dadd_rn(acc, prod); }
    static __device__ __forceinline__ V runtime_one() { return 1.0; }
};

// permutations of a warp, warps of a block (they share a tile) and samples
// copied at a time
template <class T>
constexpr int metric_q() { return sizeof(T) == 4 ? 2 : 4; }
constexpr int kMaxWarps = 8;
// resident blocks the registers are kept for
template <int ACC, class T>
constexpr int metric_blocks() {
    return sizeof(T) == 8 ? 2 : ACC == ACC_OVERKILL || ACC == ACC_KNUTH ? 3 : 4;
}
constexpr int kChunk = 32;
// class bits of a warp: a byte per sample, the chunks kPatStep bytes apart;
// behind a chunk's last pair kEnd (an odd last sample's bits follow it)
constexpr int kPatStep = kChunk + 2, kEnd = 16;
constexpr int pat_bytes(int S) { return (S + kChunk - 1) / kChunk * kPatStep; }

template <int ACC, class T>
constexpr int metric_vecs() { return sizeof(T) == 8 ? 1 : 2; }  // vectors per lane
template <int ACC, class T>
constexpr int metric_genes() { return 32 * metric_vecs<ACC, T>() * Vec<T>::kLanes; }  // genes of a tile
template <int ACC, class T>
constexpr size_t metric_smem(int warps, int S) {
    return sizeof(T) * metric_genes<ACC, T>() * (2 * kChunk + (size_t)warps) + (size_t)warps * pat_bytes(S);
}

// one copy of BYTES (4, 8, 16), both addresses aligned to it
template <int BYTES>
__device__ __forceinline__ void async_copy(uint32_t dst, const void* src) {
    if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(BYTES) : "memory");
}

// ---- the samples of the paired fp32 statistics, as one assembly loop -------
// Two samples at a time: an indirect branch on their four class bits (two
// samples, two permutations) to one of sixteen cases, each updating its
// accumulators in place.  In assembly, loop and all, because the compiler
// copies every accumulator where the cases meet (written as a C++ switch: 55
// instructions for what takes 24).  The cases never meet: each loads the next
// bits and branches on them itself, so that a pair costs 8 instructions besides
// its statistics and not 12 (20,000 genes x 200 samples x 1,000 permutations
// 944 -> 832 us).  The branch has a long latency: two vectors a lane (128 genes
// a warp) leave registers for 32 warps an SM, which hide it better than four
// vectors and 20 warps (2,000 genes x 40 samples x 1,024 43 against 54 us when
// the cases still met).
// Operand numbers: statistics of class, permutation and vector M_ 0-7, W_
// 8-15, U_ 16-23; X_ the loaded vector of a sample.
#define GM_0A0(OP) OP(0, 8, 16, 0) OP(1, 9, 17, 1)
#define GM_0A1(OP) OP(2, 10, 18, 0) OP(3, 11, 19, 1)
#define GM_0B0(OP) OP(4, 12, 20, 0) OP(5, 13, 21, 1)
#define GM_0B1(OP) OP(6, 14, 22, 0) OP(7, 15, 23, 1)
#define GM_1A0(OP) OP(0, 8, 16, 2) OP(1, 9, 17, 3)
#define GM_1A1(OP) OP(2, 10, 18, 2) OP(3, 11, 19, 3)
#define GM_1B0(OP) OP(4, 12, 20, 2) OP(5, 13, 21, 3)
#define GM_1B1(OP) OP(6, 14, 22, 2) OP(7, 15, 23, 3)
#define GM_AHEAD(PP, XP)                                                                                          \
    GM_LOAD(XP, 0, 0, 1) GM_LOAD(XP, 512, 2, 3) "ld.shared.u8 bits, [%" #PP "+2];\n"                              \
    "add.u32 %" #PP ", %" #PP ", 2;\n add.u32 %" #XP ", %" #XP ", 1024;\n"
#define GM_CASE(PP, XP, N, P0, P1, P2, P3) "C" #N ":\n" GM_AHEAD(PP, XP) P0 P1 P2 P3 "brx.idx.uni bits, TS;\n"
#define GM_CASE1(N, P0, P1) "C" #N ":\n" P0 P1 "bra.uni NEXT;\n"
#define GM_LOAD(XP, AT, A, B) "ld.shared.v2.b64 {x" #A ", x" #B "}, [%" #XP "+" #AT "];\n"
// rows of 128 genes: 512 bytes
// operands PP, XP: addresses of the class bits and of the lane's vectors; every
// case loads its samples and the next pair's bits, and branches on those; the
// bits end with kEnd
#define GM_LOOP(OP, PP, XP)                                                                                       \
    "{\n .reg .b64 d, e, x0, x1, x2, x3;\n .reg .u32 bits;\n"                                                    \
    " TS: .branchtargets C0, C1, C2, C3, C4, C5, C6, C7, C8, C9, C10, C11, C12, C13, C14, C15, OUT;\n"           \
    " ld.shared.u8 bits, [%" #PP "];\n brx.idx.uni bits, TS;\n"                                                  \
    GM_CASE(PP, XP, 0, GM_0B0(OP), GM_0B1(OP), GM_1B0(OP), GM_1B1(OP)) \
    GM_CASE(PP, XP, 1, GM_0A0(OP), GM_0B1(OP), GM_1B0(OP), GM_1B1(OP)) \
    GM_CASE(PP, XP, 2, GM_0B0(OP), GM_0A1(OP), GM_1B0(OP), GM_1B1(OP)) \
    GM_CASE(PP, XP, 3, GM_0A0(OP), GM_0A1(OP), GM_1B0(OP), GM_1B1(OP)) \
    GM_CASE(PP, XP, 4, GM_0B0(OP), GM_0B1(OP), GM_1A0(OP), GM_1B1(OP)) \
    GM_CASE(PP, XP, 5, GM_0A0(OP), GM_0B1(OP), GM_1A0(OP), GM_1B1(OP)) \
    GM_CASE(PP, XP, 6, GM_0B0(OP), GM_0A1(OP), GM_1A0(OP), GM_1B1(OP)) \
    GM_CASE(PP, XP, 7, GM_0A0(OP), GM_0A1(OP), GM_1A0(OP), GM_1B1(OP)) \
    GM_CASE(PP, XP, 8, GM_0B0(OP), GM_0B1(OP), GM_1B0(OP), GM_1A1(OP)) \
    GM_CASE(PP, XP, 9, GM_0A0(OP), GM_0B1(OP), GM_1B0(OP), GM_1A1(OP)) \
    GM_CASE(PP, XP, 10, GM_0B0(OP), GM_0A1(OP), GM_1B0(OP), GM_1A1(OP)) \
    GM_CASE(PP, XP, 11, GM_0A0(OP), GM_0A1(OP), GM_1B0(OP), GM_1A1(OP)) \
    GM_CASE(PP, XP, 12, GM_0B0(OP), GM_0B1(OP), GM_1A0(OP), GM_1A1(OP)) \
    GM_CASE(PP, XP, 13, GM_0A0(OP), GM_0B1(OP), GM_1A0(OP), GM_1A1(OP)) \
    GM_CASE(PP, XP, 14, GM_0B0(OP), GM_0A1(OP), GM_1A0(OP), GM_1A1(OP)) \
    GM_CASE(PP, XP, 15, GM_0A0(OP), GM_0A1(OP), GM_1A0(OP), GM_1A1(OP)) \
    "OUT:\n}\n"
// the last sample of an odd number
#define GM_ONE(OP, PP, XP)                                                                                        \
    "{\n .reg .b64 d, e, x0, x1;\n .reg .u32 bits;\n TS: .branchtargets C0, C1, C2, C3;\n"                        \
    " ld.shared.u8 bits, [%" #PP "];\n and.b32 bits, bits, 3;\n" GM_LOAD(XP, 0, 0, 1) " brx.idx.uni bits, TS;\n"  \
    GM_CASE1(0, GM_0B0(OP), GM_0B1(OP)) GM_CASE1(1, GM_0A0(OP), GM_0B1(OP))                                        \
    GM_CASE1(2, GM_0B0(OP), GM_0A1(OP)) GM_CASE1(3, GM_0A0(OP), GM_0A1(OP)) "NEXT:\n}\n"
// x added to the sum
#define GM_SUM(M_, W_, U_, X_) "add.rn.f32x2 %" #M_ ", %" #M_ ", x" #X_ ";\n"
// ... and x^2 to the sum of squares; one: 18
#define GM_ONEPASS(M_, W_, U_, X_)                                                        \
    GM_SUM(M_, W_, U_, X_) "mul.rn.f32x2 d, x" #X_ ", x" #X_ ";\n fma.rn.f32x2 %" #W_ ", %18, d, %" #W_ ";\n"
// Kahan step: W_ the compensation
#define GM_KAHAN(M_, W_, U_, X_)                                                                     \
    "sub.rn.f32x2 d, x" #X_ ", %" #W_ ";\n add.rn.f32x2 e, %" #M_ ", d;\n"                          \
    "sub.rn.f32x2 %" #W_ ", e, %" #M_ ";\n sub.rn.f32x2 %" #W_ ", %" #W_ ", d;\n mov.b64 %" #M_ ", e;\n"
// squared deviation from the mean M_ added to W_; one: 18
#define GM_DEV(M_, W_, U_, X_) \
    "sub.rn.f32x2 d, x" #X_ ", %" #M_ ";\n mul.rn.f32x2 d, d, d;\n fma.rn.f32x2 %" #W_ ", %18, d, %" #W_ ";\n"
// ... and the deviation itself to W_, the square to U_; one: 26
#define GM_DEV2(M_, W_, U_, X_)                                                                \
    "sub.rn.f32x2 d, x" #X_ ", %" #M_ ";\n add.rn.f32x2 %" #W_ ", %" #W_ ", d;\n"             \
    "mul.rn.f32x2 d, d, d;\n fma.rn.f32x2 %" #U_ ", %26, d, %" #U_ ";\n"
// a statistic's registers, class by class, permutation by permutation
#define GM_RW(A) "+l"(A[0][0][0]), "+l"(A[0][0][1]), "+l"(A[0][1][0]), "+l"(A[0][1][1]), "+l"(A[1][0][0]),      \
    "+l"(A[1][0][1]), "+l"(A[1][1][0]), "+l"(A[1][1][1])

enum WalkMode { WALK_SUMS, WALK_STRICT, WALK_DEVIATIONS };

// Running statistics of a lane's genes for the warp's permutations: class c
// (0: A, 1: B), permutation j, vector v.
template <int ACC, class T>
struct Stats {
    using E = Exact<T>;
    using A = Vec<T>;
    using V = typename A::V;
    static constexpr int NV = metric_vecs<ACC, T>(), L = A::kLanes, kQ = metric_q<T>();
    static constexpr bool TWO = ACC == ACC_TWOPASS || ACC == ACC_OVERKILL;
    static constexpr bool VAR = ACC == ACC_ONEPASS || ACC == ACC_KNUTH || TWO;  // variances
    static constexpr bool COMP = ACC == ACC_KAHAN || ACC == ACC_OVERKILL;       // compensated sums
    V m[2][kQ][NV];
    V q[2][COMP ? kQ : 1][COMP ? NV : 1];
    V var[2][VAR ? kQ : 1][VAR ? NV : 1];
    int it[2][ACC == ACC_KNUTH ? kQ : 1];
    V one;

    __device__ __forceinline__ void clear() {
        one = A::runtime_one();
#pragma unroll
        for (int c = 0; c < 2; c++)
#pragma unroll
            for (int j = 0; j < kQ; j++) {
                if constexpr (ACC == ACC_KNUTH) it[c][j] = 0;
#pragma unroll
                for (int v = 0; v < NV; v++) {
                    m[c][j][v] = A::zero();
                    if constexpr (COMP) q[c][j][v] = A::zero();
                    if constexpr (VAR) var[c][j][v] = A::zero();
                }
            }
    }
    // one sample with class-A bits B
    template <int MODE, int B>
    __device__ __forceinline__ void step(const V* x) {
#pragma unroll
        for (int j = 0; j < kQ; j++) {
            constexpr int kBits = B;
            const int c = ((kBits >> j) & 1) ? 0 : 1;
            if constexpr (MODE == WALK_DEVIATIONS) {
#pragma unroll
                for (int v = 0; v < NV; v++) {
                    const V d = A::sub(x[v], m[c][j][v]);
                    if constexpr (ACC == ACC_OVERKILL) q[c][j][v] = A::add(q[c][j][v], d);
                    if constexpr (TWO) var[c][j][v] = A::add_product(var[c][j][v], A::mul(d, d), one);
                }
            } else {
                if constexpr (ACC == ACC_KNUTH) it[c][j]++;
#pragma unroll
                for (int v = 0; v < NV; v++) {
                    if constexpr (COMP) {
                        const V alpha = A::sub(x[v], q[c][j][v]);
                        const V beta = A::add(m[c][j][v], alpha);
                        q[c][j][v] = A::sub(A::sub(beta, m[c][j][v]), alpha);
                        m[c][j][v] = beta;
                    } else if constexpr (ACC == ACC_KNUTH) {
                        T xs[L], ms[L], vs[L];
                        A::unpack(x[v], xs);
                        A::unpack(m[c][j][v], ms);
                        A::unpack(var[c][j][v], vs);
#pragma unroll
                        for (int l = 0; l < L; l++) {
                            const T d = E::sub(xs[l], ms[l]);
                            ms[l] = E::add(ms[l], E::div(d, (T)it[c][j]));
                            vs[l] = E::add(vs[l], E::mul(d, E::sub(xs[l], ms[l])));
                        }
                        m[c][j][v] = A::pack(ms);
                        var[c][j][v] = A::pack(vs);
                    } else {
                        m[c][j][v] = A::add(m[c][j][v], x[v]);
                        if constexpr (ACC == ACC_ONEPASS)
                            var[c][j][v] = A::add_product(var[c][j][v], A::mul(x[v], x[v]), one);
                    }
                    if constexpr (MODE == WALK_STRICT) {
                        T none[L];
#pragma unroll
                        for (int l = 0; l < L; l++) none[l] = T(0);
                        m[1 - c][j][v] = A::add(m[1 - c][j][v], A::mul(x[v], A::pack(none)));
                    }
                }
            }
        }
    }
    // whether two samples are taken by one assembly block
    template <int MODE>
    static constexpr bool paired() { return sizeof(T) == 4 && ACC != ACC_KNUTH && MODE != WALK_STRICT; }
    // the pairs of samples of a chunk (COUNT = 2) or one sample (COUNT = 1) from
    // the shared-memory addresses of their class bits and of the lane's vectors.
    // The bits are the same in every lane: one branch, no divergence.
    template <int MODE, int COUNT>
    __device__ __forceinline__ void samples(uint32_t pp, uint32_t xp) {
#define GM_RUN(OP, PP, XP, ...)                                                                                   \
    if constexpr (COUNT == 2)                                                                                     \
        asm volatile(GM_LOOP(OP, PP, XP) : __VA_ARGS__, "+r"(pp), "+r"(xp) : "l"(one) : "memory");                \
    else                                                                                                          \
        asm volatile(GM_ONE(OP, PP, XP) : __VA_ARGS__, "+r"(pp), "+r"(xp) : "l"(one) : "memory");
        if constexpr (MODE == WALK_SUMS && (ACC == ACC_NAIVE || ACC == ACC_TWOPASS)) {
            GM_RUN(GM_SUM, 8, 9, GM_RW(m))
        } else if constexpr (ACC == ACC_ONEPASS) {
            GM_RUN(GM_ONEPASS, 16, 17, GM_RW(m), GM_RW(var))
        } else if constexpr (ACC == ACC_KAHAN || (ACC == ACC_OVERKILL && MODE == WALK_SUMS)) {
            GM_RUN(GM_KAHAN, 16, 17, GM_RW(m), GM_RW(q))
        } else if constexpr (ACC == ACC_TWOPASS) {
            GM_RUN(GM_DEV, 16, 17, GM_RW(m), GM_RW(var))
        } else if constexpr (ACC == ACC_OVERKILL) {
            GM_RUN(GM_DEV2, 24, 25, GM_RW(m), GM_RW(q), GM_RW(var))
        }
#undef GM_RUN
    }
    // one sample by a switch (FP64: bound by its pipe; Knuth's divisions)
    template <int MODE>
    __device__ __forceinline__ void sample(int bits, const V* x) {
        if constexpr (kQ == 4) {
            switch (bits) {
                case 0: step<MODE, 0>(x); break;
                case 1: step<MODE, 1>(x); break;
                case 2: step<MODE, 2>(x); break;
                case 3: step<MODE, 3>(x); break;
                case 4: step<MODE, 4>(x); break;
                case 5: step<MODE, 5>(x); break;
                case 6: step<MODE, 6>(x); break;
                case 7: step<MODE, 7>(x); break;
                case 8: step<MODE, 8>(x); break;
                case 9: step<MODE, 9>(x); break;
                case 10: step<MODE, 10>(x); break;
                case 11: step<MODE, 11>(x); break;
                case 12: step<MODE, 12>(x); break;
                case 13: step<MODE, 13>(x); break;
                case 14: step<MODE, 14>(x); break;
                default: step<MODE, 15>(x); break;
            }
        } else {
            switch (bits) {
                case 0: step<MODE, 0>(x); break;
                case 1: step<MODE, 1>(x); break;
                case 2: step<MODE, 2>(x); break;
                default: step<MODE, 3>(x); break;
            }
        }
    }
};

// The expression tile of a block and its walks over the samples.
template <int ACC, class T>
struct Tile {
    using S_ = Stats<ACC, T>;
    using V = typename S_::V;
    static constexpr int NV = S_::NV, L = S_::L, GW = metric_genes<ACC, T>();
    const T* X;   // first gene of the tile
    T* tile;      // [2][kChunk][GW]
    const uint8_t* pat;
    int G, S, gn;
    bool wide;      // 16-byte copies: every row starts on a 16-byte boundary
    bool resident;  // the whole table of the tile is in the two buffers (resident())

    __device__ __forceinline__ void load(int c) const {
        constexpr int PER = 16 / (int)sizeof(T);
        const int s0 = c * kChunk, n = min(kChunk, S - s0);
        T* const to = tile + (c & 1) * kChunk * GW;
        const T* const from = X + (int64_t)s0 * G;
        // rows by warps, so that a step is one addition to either address (15,013
        // genes, copied four bytes at a time: 435 -> 377 us for the whole kernel,
        // 20,000 genes 832 -> 815)
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
        if (wide) {
            constexpr int PIECES = GW / PER, ROWS = 32 / PIECES;  // 16-byte pieces of a row, rows of a warp's copy
            const int r0 = warp * ROWS + lane / PIECES, q = lane % PIECES * PER;
            const T* src = from + (int64_t)r0 * G + q;
            uint32_t dst = smem_u32(to + r0 * GW + q);
            for (int r = r0; r < n; r += warps * ROWS) {
                async_copy<16>(dst, src);
                src += (int64_t)warps * ROWS * G;
                dst += (uint32_t)(warps * ROWS * GW * (int)sizeof(T));
            }
        } else {
            const T* src = from + (int64_t)warp * G + lane;
            uint32_t dst = smem_u32(to + warp * GW + lane);
            for (int r = warp; r < n; r += warps) {
#pragma unroll
                for (int i = 0; i < GW / 32; i++)
                    if (lane + 32 * i < gn) async_copy<(int)sizeof(T)>(dst + 32u * i * (uint32_t)sizeof(T), src + 32 * i);
                src += (int64_t)warps * G;
                dst += (uint32_t)(warps * GW * (int)sizeof(T));
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    // at most two chunks: copied once, for every pass and round of the block
    __device__ __forceinline__ void load_all() const {
        load(0);
        if (S > kChunk) load(1);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
    }
    // every sample in index order; the whole block takes part in the copies
    template <int MODE>
    __device__ __forceinline__ void walk(S_& st, bool mine) const {
        const int chunks = (S + kChunk - 1) / kChunk, lane = threadIdx.x & 31;
        if (!resident) {
            __syncthreads();  // the buffers are free
            load(0);
        }
        for (int c = 0; c < chunks; c++) {
            if (!resident) {
                if (c + 1 < chunks) {
                    load(c + 1);
                    asm volatile("cp.async.wait_group 1;" ::: "memory");
                } else {
                    asm volatile("cp.async.wait_group 0;" ::: "memory");
                }
                __syncthreads();
            }
            if (mine) {
                const int s0 = c * kChunk, n = min(kChunk, S - s0);
                const V* const row = reinterpret_cast<const V*>(tile + (c & 1) * kChunk * GW) + lane * NV;
                const uint8_t* const bits = pat + c * kPatStep;
                auto get = [&](int t, V* x) {
                    if constexpr (NV == 2) {
                        const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(row + t * (GW / L));
                        x[0] = q.x;
                        x[1] = q.y;
                    } else {
                        x[0] = row[t * (GW / L)];
                    }
                };
                if constexpr (S_::template paired<MODE>()) {
                    const uint32_t pp = smem_u32(bits), xp = smem_u32(row);
                    static_assert(GW * sizeof(T) == 512, "the loop's row stride");
                    st.template samples<MODE, 2>(pp, xp);
                    if (n & 1) st.template samples<MODE, 1>(pp + n, xp + (n - 1) * GW * (int)sizeof(T));
                } else {
#pragma unroll 1
                    for (int t = 0; t < n; t++) {
                        V x[NV];
                        get(t, x);
                        const int b = bits[sizeof(T) == 4 && t == n - 1 ? t + (n & 1) : t];
                        st.template sample<MODE>(sizeof(T) == 4 ? b & 3 : b, x);
                    }
                }
            }
            if (!resident) __syncthreads();
        }
    }
};

// One block: gene tile `gt`, permutations p0 .. p0 + kQ * warps * rounds - 1
// (a warp takes `rounds` groups one after the other; with at most two chunks
// of samples the tile is copied once for all of them).  `strict`
// (naive accumulator, a table with values that are not finite): the
// reference adds 0 * x to the other class, which is NaN there.
template <int ACC, class T>
__device__ __forceinline__ void metric_block(const T* __restrict__ X, int G, int S,
                                             const uint32_t* __restrict__ masks, int words, int num_perms, T nA, T nB,
                                             T* __restrict__ keys, int comb, bool strict, int gt, int p0, int rounds) {
    using E = Exact<T>;
    using St = Stats<ACC, T>;
    using A = Vec<T>;
    constexpr int NV = St::NV, L = St::L, GL = NV * L, GW = 32 * GL;  // vectors, genes of a lane
    constexpr int kQ = St::kQ;
    constexpr bool TWO = St::TWO, VAR = St::VAR;
    extern __shared__ __align__(16) unsigned char smem[];
    T* const tile = reinterpret_cast<T*>(smem);                 // [2][kChunk][GW]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    T* const out = tile + 2 * kChunk * GW + warp * GW;          // [warps][GW]
    uint8_t* const pat = reinterpret_cast<uint8_t*>(tile + (2 * kChunk + warps) * GW) + warp * pat_bytes(S);  // [warps]
    const int g0 = gt * GW;
    const int gn = min(GW, G - g0);  // genes of the tile
    const bool wide = gn == GW && (G % (16 / (int)sizeof(T))) == 0 && (reinterpret_cast<uintptr_t>(X) & 15u) == 0;
    const Tile<ACC, T> tl{X + g0, tile, pat, G, S, gn, wide, S <= 2 * kChunk};
    if (tl.resident) tl.load_all();

    for (int round = 0; round < rounds; round++) {
        const int p = p0 + (round * warps + warp) * kQ;  // the warp's permutations
        const bool mine = p < num_perms;
        __syncwarp();
        if (mine) {  // class-A bits of the permutations, a byte per sample; above them the next sample's
            for (int w = 0; w < words; w++) {
                uint32_t mw[kQ], b = 0u;
#pragma unroll
                for (int j = 0; j < kQ; j++) {
                    mw[j] = p + j < num_perms ? __ldg(masks + (int64_t)(p + j) * words + w) : 0u;
                    b |= ((mw[j] >> lane) & 1u) << j;
                }
                if (sizeof(T) == 4) b |= __shfl_down_sync(kFullMask, b, 1) << kQ;  // pairs start at even samples
                const int n = min(kChunk, S - w * 32);
                uint8_t* const to = pat + w * kPatStep;
                if (sizeof(T) == 4 && lane == 0) to[n & ~1] = kEnd;
                if (lane < n) to[sizeof(T) == 4 && lane == n - 1 ? lane + (n & 1) : lane] = (uint8_t)b;
            }
        }
        __syncwarp();
        St st;
        st.clear();
        // pass 1: sums (or running means and squares)
        if constexpr (ACC == ACC_NAIVE) {
            if (strict) tl.template walk<WALK_STRICT>(st, mine);
            else tl.template walk<WALK_SUMS>(st, mine);
        } else {
            tl.template walk<WALK_SUMS>(st, mine);
        }
        const ClassSize<T> n[2] = {ClassSize<T>(nA), ClassSize<T>(nB)};
#pragma unroll
        for (int c = 0; c < 2; c++)
#pragma unroll
            for (int j = 0; j < kQ; j++)
#pragma unroll
                for (int v = 0; v < NV; v++) {
                    T ms[L], vs[L];
                    A::unpack(st.m[c][j][v], ms);
                    if constexpr (VAR) A::unpack(st.var[c][j][v], vs);
#pragma unroll
                    for (int l = 0; l < L; l++) {
                        if constexpr (ACC != ACC_KNUTH) ms[l] = n[c].divides(ms[l]);
                        if constexpr (ACC == ACC_ONEPASS) vs[l] = E::sub(n[c].divides(vs[l]), E::mul(ms[l], ms[l]));
                        if constexpr (ACC == ACC_KNUTH) vs[l] = n[c].divides(vs[l]);
                    }
                    st.m[c][j][v] = A::pack(ms);
                    if constexpr (VAR && !TWO) st.var[c][j][v] = A::pack(vs);
                    if constexpr (ACC == ACC_OVERKILL) st.q[c][j][v] = A::zero();  // sums of deviations from here on
                }
        // pass 2: squared deviations from the own class mean
        if constexpr (TWO) tl.template walk<WALK_DEVIATIONS>(st, mine);
        if (!mine) continue;
        // the metric, its keys stored a permutation at a time
#pragma unroll
        for (int j = 0; j < kQ; j++) {
            if (p + j >= num_perms) break;
            T key[GL];
#pragma unroll
            for (int v = 0; v < NV; v++) {
                T ms[2][L], vs[2][L], qs[L];
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    A::unpack(st.m[c][j][v], ms[c]);
                    if constexpr (VAR) A::unpack(st.var[c][j][v], vs[c]);
                    if constexpr (ACC == ACC_OVERKILL) {
                        A::unpack(st.q[c][j][v], qs);
#pragma unroll
                        for (int l = 0; l < L; l++) vs[c][l] = E::sub(vs[c][l], n[c].divides(E::mul(qs[l], qs[l])));
                    }
#pragma unroll
                    for (int l = 0; l < L; l++) {
                        if constexpr (TWO) vs[c][l] = n[c].divides(vs[c][l]);
                        if constexpr (!VAR) vs[c][l] = T(0);
                    }
                }
#pragma unroll
                for (int l = 0; l < L; l++)
                    key[v * L + l] = canonical_nan(combine<T>(comb, ms[0][l], vs[0][l], n[0], ms[1][l], vs[1][l], n[1]));
            }
#pragma unroll
            for (int i = 0; i < GL; i++) out[lane * GL + i] = key[i];
            __syncwarp();
            T* const kp = keys + (int64_t)(p + j) * G + g0;
#pragma unroll
            for (int i = 0; i < GL; i++)
                if (lane + 32 * i < gn) kp[lane + 32 * i] = out[lane + 32 * i];
            __syncwarp();
        }
    }
}

template <int ACC, class T>
__global__ void __launch_bounds__(32 * kMaxWarps, metric_blocks<ACC, T>())
metric_kernel(const T* __restrict__ X, int G, int S, const uint32_t* __restrict__ masks, int words, int num_perms,
              T nA, T nB, T* __restrict__ keys, int comb, const int* __restrict__ finite, int rounds) {
    const bool strict = ACC == ACC_NAIVE && finite && *finite == 0;
    metric_block<ACC, T>(X, G, S, masks, words, num_perms, nA, nB, keys, comb, strict, blockIdx.x,
                         blockIdx.y * (blockDim.x >> 5) * metric_q<T>() * rounds, rounds);
}

// every instance of a batch group in one launch (blockIdx.z = instance; the
// grid covers the largest instance, blocks beyond an instance's extent leave)
template <int ACC, class T>
__global__ void __launch_bounds__(32 * kMaxWarps, metric_blocks<ACC, T>())
metric_multi(const MetricTask<T>* __restrict__ tasks, int comb, int rounds) {
    const MetricTask<T> t = tasks[blockIdx.z];
    const int p0 = blockIdx.y * (blockDim.x >> 5) * metric_q<T>() * rounds;
    if ((int)blockIdx.x * metric_genes<ACC, T>() >= t.G || p0 >= t.num_perms) return;
    const bool strict = ACC == ACC_NAIVE && t.fast_ok && *t.fast_ok == 0;
    metric_block<ACC, T>(t.X, t.G, t.S, t.masks, t.words, t.num_perms, t.nA, t.nB, t.keys, comb, strict, blockIdx.x,
                         p0, rounds);
}

inline int metric_sms() {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
}

// Warps of a block: eight share a tile; fewer where that leaves SMs without
// two blocks (few permutations of few genes; `units`: gene tiles times groups
// of a warp), or where the class bits of very many samples need the shared
// memory.  The grid's second dimension (at most 65,535 blocks) is a batch's
// groups by the warps of a block.
constexpr int kMetricMaxPerms = 4 * 65535;
template <int ACC, class T>
int metric_warps(int64_t units, int64_t groups, int S) {
    const int64_t want = 2 * (int64_t)metric_sms();
    int w = kMaxWarps;
    while (w > 1 && (units / w < want || metric_smem<ACC, T>(w, S) > 110 * 1024) &&
           (groups + w / 2 - 1) / (w / 2) <= 65535)
        w >>= 1;
    return w;
}

// Rounds of a warp: as tuned, but in fp32 where the tile stays in shared memory
// two, if that leaves some sixteen blocks an SM: the copies once for both.  More
// rounds make long blocks and an uneven end: onepass T test, 7,411 genes x 57 x
// 2,000, 1, 2, 4, 8 rounds 159, 153, 158, 169 us; two-pass signal to noise, 20,000
// x 40 x 1,000, 245, 237, 252, 271; log2 ratio, 60,963 x 16 x 338, 130, 133, 140, 155.
// fp64 waits for its pipe and not for the copies: difference of classes, 20,000 x
// 60 x 400, 1,196, 1,254, 1,338, 1,426.
template <int ACC, class T>
int metric_rounds(int64_t tiles, int64_t num_perms, int S, int tuned) {
    if (sizeof(T) == 8 || S > 2 * kChunk) return tuned;
    const int64_t blocks = tiles * num_perms / (metric_q<T>() * kMaxWarps);
    const int64_t r = blocks / (16 * (int64_t)metric_sms());
    return r < tuned ? tuned : r > 2 ? 2 : (int)r;
}

template <int ACC, class T>
cudaError_t launch_metric_acc(int comb, const T* X, int G, int S, const uint32_t* masks, int words, int num_perms,
                              int64_t nA, int64_t nB, T* keys, const int* finite, int tuned, cudaStream_t st) {
    const int tiles = (G + metric_genes<ACC, T>() - 1) / metric_genes<ACC, T>();
    const int rounds = metric_rounds<ACC, T>(tiles, num_perms, S, tuned);
    const int per = metric_q<T>() * rounds, groups = (num_perms + per - 1) / per;
    const int w = metric_warps<ACC, T>((int64_t)tiles * groups, groups, S);
    const size_t smem = metric_smem<ACC, T>(w, S);
    auto kern = metric_kernel<ACC, T>;
    if (smem > 48 * 1024) {
        cudaError_t e = allow_smem(kern, smem);
        if (e != cudaSuccess) return e;
    }
    kern<<<dim3((unsigned)tiles, (unsigned)((groups + w - 1) / w)), 32 * w, smem, st>>>(
        X, G, S, masks, words, num_perms, (T)nA, (T)nB, keys, comb, finite, rounds);
    launches_add(1);
    return cudaGetLastError();
}

// accumulator and combiner of a metric id
inline bool metric_parts(int metric, int& acc, int& comb) {
    static const int accs[14] = {ACC_NAIVE, ACC_NAIVE, ACC_NAIVE, ACC_KAHAN, ACC_KAHAN, ACC_KAHAN, ACC_ONEPASS,
                                 ACC_ONEPASS, ACC_TWOPASS, ACC_TWOPASS, ACC_KNUTH, ACC_KNUTH, ACC_OVERKILL,
                                 ACC_OVERKILL};
    static const int combs[14] = {COMB_DIFF, COMB_RATIO, COMB_LOG2, COMB_DIFF, COMB_RATIO, COMB_LOG2, COMB_S2N,
                                  COMB_TTEST, COMB_S2N, COMB_TTEST, COMB_S2N, COMB_TTEST, COMB_S2N, COMB_TTEST};
    if (metric < 0 || metric >= 14) return false;
    acc = accs[metric];
    comb = combs[metric];
    return true;
}

#define GSEA_BY_ACC(CALL)                      \
    switch (acc) {                             \
        case ACC_NAIVE: CALL(ACC_NAIVE);       \
        case ACC_KAHAN: CALL(ACC_KAHAN);       \
        case ACC_ONEPASS: CALL(ACC_ONEPASS);   \
        case ACC_TWOPASS: CALL(ACC_TWOPASS);   \
        case ACC_KNUTH: CALL(ACC_KNUTH);       \
        default: CALL(ACC_OVERKILL);           \
    }

// pb: rounds of a warp, 4 (0): one, 8: two; identical keys
template <class T>
cudaError_t launch_metric_impl(int metric, const T* X, int G, int S, const uint32_t* masks, int words, int num_perms,
                               int64_t nA, int64_t nB, T* keys, const int* finite, cudaStream_t st, int pb) {
    int acc, comb;
    if ((pb != 0 && pb != 4 && pb != 8) || !metric_parts(metric, acc, comb)) return cudaErrorInvalidValue;
    if (num_perms <= 0) return cudaSuccess;
    if (num_perms > kMetricMaxPerms) return cudaErrorInvalidValue;
#define GSEA_CALL(A) \
    return launch_metric_acc<A, T>(comb, X, G, S, masks, words, num_perms, nA, nB, keys, finite, pb == 8 ? 2 : 1, st)
    GSEA_BY_ACC(GSEA_CALL)
#undef GSEA_CALL
}

// Batched instances: the group key of an instance (instances with equal keys
// share one launch): the metric and the rounds of a warp.
inline int metric_multi_key_impl(int metric, int pb) { return metric * 2 + (pb == 8 ? 1 : 0); }

template <int ACC, class T>
cudaError_t launch_metric_multi_acc(int comb, int rounds, const MetricTask<T>* d, const MetricTask<T>* h, int n,
                                    cudaStream_t st) {
    int64_t tiles = 1, groups = 1, work = 0;
    int smax = 0;
    for (int i = 0; i < n; i++) {
        const int64_t t = (h[i].G + metric_genes<ACC, T>() - 1) / metric_genes<ACC, T>();
        const int per = metric_q<T>() * rounds;
        const int64_t g = (h[i].num_perms + per - 1) / per;
        tiles = std::max(tiles, t);
        groups = std::max(groups, g);
        work += t * g;
        smax = std::max(smax, h[i].S);
    }
    const int w = metric_warps<ACC, T>(work, groups, smax);
    const size_t smem = metric_smem<ACC, T>(w, smax);
    auto kern = metric_multi<ACC, T>;
    if (smem > 48 * 1024) {
        cudaError_t e = allow_smem(kern, smem);
        if (e != cudaSuccess) return e;
    }
    kern<<<dim3((unsigned)tiles, (unsigned)((groups + w - 1) / w), (unsigned)n), 32 * w, smem, st>>>(d, comb, rounds);
    launches_add(1);
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_metric_multi_impl(int key, const MetricTask<T>* d, const MetricTask<T>* h, int n,
                                     cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    if (n > 65535) return cudaErrorInvalidValue;
    for (int i = 0; i < n; i++)
        if (h[i].num_perms > kMetricMaxPerms) return cudaErrorInvalidValue;
    int acc, comb;
    if (!metric_parts(key / 2, acc, comb)) return cudaErrorInvalidValue;
#define GSEA_CALL(A) return launch_metric_multi_acc<A, T>(comb, key % 2 + 1, d, h, n, st)
    GSEA_BY_ACC(GSEA_CALL)
#undef GSEA_CALL
}
#undef GSEA_BY_ACC

}  // namespace gsea
