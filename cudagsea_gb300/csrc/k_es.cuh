// k_es.cuh -- enrichment scores for gene sets x permutations (included by
// k_es_f32.cu and k_es_f64.cu, one translation unit per precision).
//
// The reference (score_kernel_shared, src/include/enrichment_scores.cuh:91-206)
// walks the whole ranked list of every (set, permutation) twice: pass 1 sums
// N_R = sum |metric| over hits and counts N_H, pass 2 runs the Kahan running
// sum (hit: +|metric|/N_R, miss: -1/(G-N_H)) and keeps the first value of
// largest magnitude, sign included.  That is K*P*G*2 steps.
//
// Here the running sum is evaluated in closed form at its only possible
// extrema: just before and just after each hit (the sum falls monotonically
// between hits).  With hits at positions r_1 < ... < r_n, weights w_j and
// m_j = r_j - (j-1) misses before hit j:
//     before hit j:  W_{j-1}/N_R - m_j * d        (position r_j - 1)
//     after  hit j:  W_j    /N_R - m_j * d        (position r_j)
//     end of list :  W_n    /N_R - (G-n) * d      (position G-1)
// with W_j the prefix sum of weights in rank order and d = (T)(1/(G-N_H)) the
// reference's decay.  The winner is the largest |value|, earliest position on
// ties, exactly the reference's strict `|Res| > |Bsf|` update; NaN weights
// propagate the same way (the reference's Res stays NaN after the first NaN
// step, and so does every later candidate here).
//
// Work per (set, permutation) is O(G/32 + n) instead of O(G):
//   * one CTA per permutation stages the rank of every gene and the weight at
//     every position in shared memory (or, when the bitmaps of large G leave
//     no room, the ranks only, the weights then read through L1 / L2);
//   * a warp takes the next set from a CTA-wide counter (largest sets first),
//     marks its members' ranks in a per-warp bitmap and sums the weights of
//     the marked ranks (N_R).  The members come from lists laid out at upload
//     (es_lists_kernel): 16-bit gene ids, a lane's four members of a group of
//     128 in one 8-byte load, no bounds or duplicate checks left to make;
//   * each lane owns a contiguous range of bitmap words: their popcounts and
//     one warp scan give the global index of the lane's first hit, and the
//     lane walks its hits once, in rank order, with a lane-local prefix of the
//     weights; its largest and smallest candidates are shifted afterwards by
//     the weight of the hits before the lane (a second warp scan);
//   * two integer warp reductions give the largest and the smallest value.
//   With 32-bit ranks (G > 65,536) a general procedure walks each lane's
//   word range twice from shared memory instead.
//
// Rounding: fp32 sums are compensated (Kahan in a lane, float-float across
// lanes), so the fp32 ES stay within a few ulp of the reference's Kahan
// running sum (the shift adds one rounding).  fp64: the walk runs in fp32 and
// only finds where the extremum is; the score there is then evaluated from
// double sums over the set's members.  Where fp32 cannot tell which hit (or
// which sign) wins, the set is walked again in double throughout (20,000 genes,
// 1,000 sets x 1,000 permutations: 7,978 us walked in double, where the FP64
// pipe takes 80 cycles an instruction, 2,890 so, where it waits for the double
// weights, a sector each from L2).
//
// What bounds it: issue slots (1,000 sets x 1,000 permutations at 20,000
// genes, fp32).  The walk is the largest part, 14 trips of the longest lane
// for 8 hits per lane, so the trips carry as little as possible: bitmap words
// hold the lowest rank in their top bit (one leading-zero count finds it, no
// bit reversal), positions and miss counts are kept times four (byte offsets
// of the weights; the decay is divided by four, exactly), the miss count
// becomes a float by an addition instead of a conversion, the extrema carry
// no positions and the words are cleared afterwards, 16 bytes at a time.
// Positions decide a score only when the largest and the smallest value have
// the same magnitude: such a set, and one whose weights are not finite, takes
// the procedure with positions (set_score_positions).
#pragma once
#include <algorithm>
#include <climits>
#include <type_traits>

#include <math_constants.h>

#include "common.cuh"
#include "kernels.h"

namespace gsea {
namespace {

// compensated accumulator: float-float for fp32, plain double for fp64
template <class T> struct Acc;
template <> struct Acc<float> {
    float hi = 0.f, lo = 0.f;
    // Kahan step (the running sum of one lane grows monotonically)
    __device__ __forceinline__ void add(float b) {
        const float y = __fsub_rn(b, lo);
        const float t = __fadd_rn(hi, y);
        lo = __fsub_rn(__fsub_rn(t, hi), y);
        hi = t;
    }
    // merge another accumulator: two-sum of the main terms, the rounding
    // error folded into the (negated) compensation
    __device__ __forceinline__ void merge(const Acc& o) {
        const float s = __fadd_rn(hi, o.hi);
        const float bb = __fsub_rn(s, hi);
        const float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bb)), __fsub_rn(o.hi, bb));
        hi = s;
        lo = __fsub_rn(__fadd_rn(lo, o.lo), err);
    }
    __device__ __forceinline__ float value() const { return __fsub_rn(hi, lo); }
    // (hi - lo) * inv + c, with one rounding of the product's main term
    __device__ __forceinline__ float scaled_plus(float inv, float c) const {
        return fmaf(hi, inv, fmaf(-lo, inv, c));
    }
    __device__ __forceinline__ Acc shfl_up(int o) const {
        Acc r;
        r.hi = __shfl_up_sync(kFullMask, hi, o);
        r.lo = __shfl_up_sync(kFullMask, lo, o);
        return r;
    }
    __device__ __forceinline__ Acc shfl_xor(int o) const {
        Acc r;
        r.hi = __shfl_xor_sync(kFullMask, hi, o);
        r.lo = __shfl_xor_sync(kFullMask, lo, o);
        return r;
    }
};
template <> struct Acc<double> {
    double hi = 0.0, lo = 0.0;  // lo unused
    __device__ __forceinline__ void add(double b) { hi += b; }
    __device__ __forceinline__ void merge(const Acc& o) { hi += o.hi; }
    __device__ __forceinline__ double value() const { return hi; }
    __device__ __forceinline__ double scaled_plus(double inv, double c) const { return fma(hi, inv, c); }
    __device__ __forceinline__ Acc shfl_up(int o) const {
        Acc r;
        r.hi = __shfl_up_sync(kFullMask, hi, o);
        return r;
    }
    __device__ __forceinline__ Acc shfl_xor(int o) const {
        Acc r;
        r.hi = __shfl_xor_sync(kFullMask, hi, o);
        return r;
    }
};

// candidate (val, pos) replaces (best, bpos) when |val| > |best|, or equal
// magnitude at an earlier position; NaN never replaces
template <class T>
__device__ __forceinline__ void consider(T val, int pos, T& best, int& bpos) {
    const T a = fabs(val), b = fabs(best);
    if (a > b || (a == b && pos < bpos)) {
        best = val;
        bpos = pos;
    }
}

// ---------------------------------------------------------------------------
// Per-set procedures.  All run on one warp with the set's member ranks marked
// in the warp's bitmap `bm` (G bits): rank r in word r / 32.  The direct
// procedures (G <= 1024*WPL) keep rank r in bit 31 - r % 32, and their words
// are cleared by clear_words; the general one keeps it in bit r % 32 and
// leaves the bitmap all zero.

// order-preserving signed 64-bit key of a double (an involution): the
// integer order of the keys is the numeric order of non-NaN doubles, -0
// below +0
__device__ __forceinline__ long long okey(double v) {
    const long long b = __double_as_longlong(v);
    return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}
__device__ __forceinline__ double okey_value(long long k) {
    return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffll));
}

// A lane's words are read and cleared 16 bytes at a time, eight lanes at
// once: where the lanes' regions lie a multiple of 64 or 128 bytes apart (WPL
// 16, 32, 48, 64) they meet in the same banks (4- and 8-way; two thirds of
// the time of a set at 60,000 genes), so those regions are 16 bytes longer.
template <int WPL>
__host__ __device__ constexpr int lane_stride() { return WPL > 0 && WPL % 16 == 0 ? WPL + 4 : WPL; }
// the bitmap word of rank r
template <int WPL>
__device__ __forceinline__ uint32_t* rank_word(uint32_t* bm, uint32_t r) {
    const uint32_t w = r >> 5;
    return bm + (lane_stride<WPL>() == WPL ? w : w + 4u * (w / (uint32_t)(WPL > 0 ? WPL : 1)));
}

// bit i from the top of a word, and the place from the top of a word's
// highest bit (nonzero words: one instruction, where a count of leading zeros
// also has to answer for zero)
__device__ __forceinline__ uint32_t top_bit(int i) { return 0x80000000u >> i; }
__device__ __forceinline__ int top_place(uint32_t v) {
    int i;
    asm("bfind.shiftamt.u32 %0, %1;" : "=r"(i) : "r"(v));
    return i;
}

// A lane's share of the bitmap: words w0 .. w0 + WPL - 1 (w0 = lane*WPL).
// nz marks its nonzero words, word i in bit 31 - i (words from 32 on in nz2).
template <int WPL>
struct LaneWords {
    uint32_t nz = 0u, nz2 = 0u;
    int cnt = 0;
    __device__ __forceinline__ explicit LaneWords(const uint32_t* bmw) {
#pragma unroll
        for (int i = 0; i < WPL; i += 4) {
            const uint4 v = *reinterpret_cast<const uint4*>(bmw + i);
            // four counts (at most 32 each) in the bytes of a word: summed at
            // once, and turned into four marks (bit 7 of a byte plus 127 says
            // the count is not zero; the product gathers bits 7, 15, 23, 31)
            const uint32_t c = ((uint32_t)__popc(v.x) << 24) + ((uint32_t)__popc(v.y) << 16) +
                               ((uint32_t)__popc(v.z) << 8) + (uint32_t)__popc(v.w);
            cnt = (int)__dp4a(c, 0x01010101u, (uint32_t)cnt);
            const uint32_t m = ((((c + 0x7f7f7f7fu) & 0x80808080u) * 0x204081u) & 0xf0000000u) >> (i & 31);
            if (i < 32) nz |= m; else nz2 |= m;
        }
    }
};
template <int WPL>
__device__ __forceinline__ void clear_words(uint32_t* bmw) {
#pragma unroll
    for (int i = 0; i < WPL; i += 4) *reinterpret_cast<uint4*>(bmw + i) = make_uint4(0u, 0u, 0u, 0u);
}

// the lane's hits in rank order: next() gives four times the rank.  The step
// to the lane's next nonzero word (taken by some lane at nearly every hit) is
// predicated instead of branched around.
template <int WPL>
struct HitWalk {
    uint32_t bmw;  // shared-memory address of the lane's words
    uint32_t nz, nz2, cur = 0u;
    uint32_t word4 = 0u, lane4;  // four times the rank of the word's top bit / of the lane's first
    __device__ __forceinline__ HitWalk(const uint32_t* words, int w0, const LaneWords<WPL>& w)
        : bmw((uint32_t)__cvta_generic_to_shared(words)), nz(w.nz), nz2(w.nz2), lane4((uint32_t)w0 << 7) {}
    // next()'s reads are unknown to the compiler, which could move the clearing
    // of the words before them: every store after the walk's scope stays behind
    // this, and its inputs are what the last read gave
    __device__ __forceinline__ ~HitWalk() { asm volatile("" ::"r"(cur), "r"(nz) : "memory"); }
    __device__ __forceinline__ uint32_t next() {
        if (WPL > 32 && (cur | nz) == 0u) {
            nz = nz2;
            bmw += 32u * 4u;
            lane4 += 32u << 7;
        }
        // No memory clobber, which would order the walk's other loads too: the
        // words were marked before nz was read from them, and are cleared after
        // the walk's scope (the destructor).
        asm(
            "{\n"
            " .reg .pred p;\n"
            " .reg .u32 i, t, a;\n"
            " setp.eq.u32 p, %0, 0;\n"
            " @p bfind.shiftamt.u32 i, %1;\n"
            " @p shr.u32 t, 0x80000000, i;\n"
            " @p xor.b32 %1, %1, t;\n"
            " @p mad.lo.u32 a, i, 4, %3;\n"
            " @p ld.shared.u32 %0, [a];\n"
            " @p mad.lo.u32 %2, i, 128, %4;\n"
            "}"
            : "+r"(cur), "+r"(nz), "+r"(word4)
            : "r"(bmw), "r"(lane4));
        const int bit = top_place(cur);
        cur ^= top_bit(bit);
        return word4 + ((uint32_t)bit << 2);
    }
};

template <class T>
__device__ __forceinline__ T weight_at(const T* wt, uint32_t r4) {
    return *reinterpret_cast<const T*>(reinterpret_cast<const char*>(wt) + (size_t)r4 * (sizeof(T) / 4));
}

// exclusive count of the hits in the lanes before, and their total n
__device__ __forceinline__ int hits_before(int cnt, int lane, int& n) {
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFullMask, incl, o);
        if (lane >= o) incl += y;
    }
    n = __shfl_sync(kFullMask, incl, 31);
    return incl - cnt;
}
// weight of the hits in the lanes before, times inv (0 where there is none)
template <class T>
__device__ __forceinline__ T weight_before(const Acc<T>& Wl, int excl, T inv, int lane) {
    Acc<T> W_incl = Wl;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const Acc<T> y = W_incl.shfl_up(o);
        if (lane >= o) W_incl.merge(y);
    }
    const Acc<T> W_pre = W_incl.shfl_up(1);
    return excl > 0 ? W_pre.scaled_plus(inv, T(0)) : T(0);
}

// Procedure with positions (any weights): every lane walks its hits once and
// keeps its largest value after a hit (mx at pmx) and smallest before one (mn
// at pmn) with the lane-local prefix Wl; the weight of the lanes before
// shifts both by a constant, which leaves their positions unchanged.  The
// set's total weight Wt (every lane) comes from the marking.  fp64 with
// finite candidates compares them as integer keys, on the integer pipe
// instead of the FP64 pipe (the keys order finite doubles as they compare
// except -0 / +0, and a zero never decides a score).
template <class T, int WPL>
__device__ __forceinline__ T set_score_positions(const uint32_t* bmw, int w0, const T* wt,
                                                 const T* __restrict__ decay, int G, int lane, const Acc<T>& Wt) {
    const LaneWords<WPL> words(bmw);
    int n;
    const int excl = hits_before(words.cnt, lane, n);
    const T inv = n > 0 ? T(1) / Wt.value() : T(0);
    const T d = decay[n];
    Acc<T> Wl;
    T mx = -CUDART_INF, mn = CUDART_INF;
    int pmx = -1, pmn = -1;
    bool ikey = false;
    long long kmx = 0, kmn = 0;
    if constexpr (std::is_same<T, double>::value) {
        ikey = isfinite(Wt.value()) && isfinite(inv);  // every candidate is finite
        kmx = okey(mx);
        kmn = okey(mn);
    }
    HitWalk<WPL> hit(bmw, w0, words);
    for (int t = 0; t < words.cnt; t++) {
        const uint32_t r4 = hit.next();
        const int r = (int)(r4 >> 2);
        const T md = -(T)(r - (excl + t)) * d;  // misses before this hit, times the decay
        const T before = t > 0 ? Wl.scaled_plus(inv, md) : md;
        Wl.add(weight_at(wt, r4));
        const T after = Wl.scaled_plus(inv, md);
        if constexpr (std::is_same<T, double>::value) {
            if (ikey) {
                const long long kb = okey(before), ka = okey(after);
                if (kb < kmn) { kmn = kb; pmn = r - 1; }
                if (ka > kmx) { kmx = ka; pmx = r; }
                continue;
            }
        }
        if (before < mn) { mn = before; pmn = r - 1; }
        if (after > mx) { mx = after; pmx = r; }
    }
    if constexpr (std::is_same<T, double>::value) {
        if (ikey) {
            mx = okey_value(kmx);
            mn = okey_value(kmn);
        }
    }
    const T shift = weight_before<T>(Wl, excl, inv, lane);
    mx += shift;
    mn += shift;
    if (lane == 31) {  // end of the list, after the trailing misses
        const T tail = -(T)(G - n) * d;
        const T end = n > 0 ? Wt.scaled_plus(inv, tail) : tail;
        if (end < mn) { mn = end; pmn = G - 1; }
    }
    // the largest value is always just after a hit and the smallest just
    // before one (or at the end): only a positive maximum and a negative
    // minimum are candidates
    T best = T(0);
    int bpos = -1;
    if (pmx >= 0 && mx > T(0)) consider<T>(mx, pmx, best, bpos);
    if (pmn >= 0 && mn < T(0)) consider<T>(mn, pmn, best, bpos);
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        const T ob = __shfl_xor_sync(kFullMask, best, o);
        const int op = __shfl_xor_sync(kFullMask, bpos, o);
        consider<T>(ob, op, best, bpos);
    }
    return best;
}

template <int WPL>  // out of line: seldom taken
__device__ __noinline__ float set_score_positions_f32(const uint32_t* bmw, int w0, const float* wt,
                                                      const float* __restrict__ decay, int G, int lane,
                                                      Acc<float> Wt) {
    return set_score_positions<float, WPL>(bmw, w0, wt, decay, G, lane, Wt);
}

// largest positive / most negative value over the warp as bits of their
// magnitudes (0 where there is none): non-negative floats order as integers
__device__ __forceinline__ uint32_t warp_top(float v) {
    return __reduce_max_sync(kFullMask, __float_as_uint(fmaxf(v, 0.f)));
}

// fp32, direct procedure: the values of set_score_positions without the
// positions, which decide nothing unless the two extrema tie in magnitude.
// Every operation on the values is the same, so the scores are the same bits:
// the miss count times four is exact and so is d / 4, and with hi = lo = 0
// the first hit's `before` is md itself for a finite inv.
template <int WPL>
__device__ __forceinline__ float set_score_direct(const uint32_t* bmw, int w0, const float* wt,
                                                  const float* __restrict__ decay, int G, int lane,
                                                  const Acc<float>& Wt) {
    const LaneWords<WPL> words(bmw);
    int n;
    const int excl = hits_before(words.cnt, lane, n);
    const float inv = n > 0 ? 1.f / Wt.value() : 0.f;
    const float d = decay[n];
    if (__all_sync(kFullMask, isfinite(Wt.value()) && isfinite(inv))) {
        const float d4 = 0.25f * d;
        constexpr uint32_t kMagic = 0x4b000000u;  // 2^23: adding a count below 2^23 to its bits adds it to its value
        uint32_t e4 = 4u * (uint32_t)excl - kMagic;
        const uint32_t end4 = e4 + 4u * (uint32_t)words.cnt;
        Acc<float> Wl;
        float mx = -CUDART_INF_F, mn = CUDART_INF_F;
        HitWalk<WPL> hit(bmw, w0, words);
#pragma unroll 2  // the sums change registers at every hit: two hits need no moves
        while (e4 != end4) {
            const uint32_t r4 = hit.next();
            const float m4 = __fadd_rn(__uint_as_float(r4 - e4), -8388608.f);  // misses before this hit, times 4
            const float md = __fmul_rn(-m4, d4);
            mn = fminf(mn, Wl.scaled_plus(inv, md));
            Wl.add(weight_at(wt, r4));
            mx = fmaxf(mx, Wl.scaled_plus(inv, md));
            e4 += 4u;
        }
        const float shift = weight_before<float>(Wl, excl, inv, lane);
        mx += shift;
        mn += shift;
        if (lane == 31) {  // end of the list, after the trailing misses
            const float tail = -(float)(G - n) * d;
            mn = fminf(mn, n > 0 ? Wt.scaled_plus(inv, tail) : tail);
        }
        const uint32_t up = warp_top(mx), down = warp_top(-mn);
        if (up > down) return __uint_as_float(up);  // warp-uniform
        if (down > up) return -__uint_as_float(down);
        if (up == 0u) return 0.f;
    }
    return set_score_positions_f32<WPL>(bmw, w0, wt, decay, G, lane, Wt);
}

// fp64 where fp32 cannot decide: the set's weight from its list (a member to
// a lane at a time, in the list's order, four gathers in flight; walking the
// marked ranks for it took as long as a third of the procedure), then the
// procedure with positions in double.  A weight that is NaN leaves one finite
// value, the one before the first hit: no walk (sets of a table with absent
// genes under the ratios and signal to noise: 200 sets x 400 permutations of
// 20,000 genes of low counts 905 -> 223 us).  Out of line: seldom taken.
template <int WPL>
__device__ __noinline__ double set_score_positions_f64(const uint32_t* bmw, int w0, const double* wt,
                                                       const uint16_t* rk, const uint2* list, int n,
                                                       const double* __restrict__ decay, int G, int lane) {
    Acc<double> Wt;
    uint32_t first = 0xffffffffu;
    for (int base = 0; base < n; base += 128, list += 32) {
        const uint2 q = __ldg(list);
        const uint32_t g[4] = {q.x & 0xffffu, q.x >> 16, q.y & 0xffffu, q.y >> 16};
        uint32_t r[4];
        double a[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {  // entries behind the last member are valid ids
            r[i] = rk[g[i]];
            a[i] = wt[r[i]];
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (base + 32 * i + lane < n) {
                Wt.add(a[i]);
                first = min(first, r[i]);
            }
        }
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) Wt.merge(Wt.shfl_xor(o));
    if (Wt.value() != Wt.value()) {  // the same in every lane
        first = __reduce_min_sync(kFullMask, first);
        return first > 0u ? -(double)first * decay[n] : 0.0;
    }
    return set_score_positions<double, WPL>(bmw, w0, wt, decay, G, lane, Wt);
}

// fp64, direct procedure: the walk in fp32, to find the hit the score is
// taken at; no fp32 value enters the score.  A candidate here is off by less
// than 10 roundings of 2^-24, 6e-7: of the weights, their compensated sum, its
// reciprocal (two), the product, the decay, the misses times it, their sum and
// the shift by the lanes before, of values at most 1.  An extremum ahead of
// every other candidate by kMargin, three times what two of them can be off, is
// the extremum.  The scores are as exact as those of the walk in double, or more
// so, having fewer roundings: against 128-bit sums over 2,000 to 60,000 genes
// 5.0e-17 rms and 2.4e-16 at most, 7.4e-17 and 3.4e-16 walked in double.  Returns the rank of the
// hit (the largest value: after it, the smallest: before it), or -1 where the
// lead is smaller, the end of the list would win, or the weights are outside
// fp32's range.  `wf(r4)`: the weight at rank r4 / 4 as a float.
constexpr float kMargin = 4e-6f;
template <int WPL, class Weight>
__device__ __forceinline__ int find_extremum(const uint32_t* bmw, int w0, Weight&& wf,
                                             const double* __restrict__ decay, int G, int lane,
                                             const Acc<float>& Wt, int& n, bool& largest) {
    const LaneWords<WPL> words(bmw);
    const int excl = hits_before(words.cnt, lane, n);
    const float inv = n > 0 ? 1.f / Wt.value() : 0.f;
    largest = false;
    if (!__all_sync(kFullMask, isfinite(Wt.value()) && isfinite(inv) && Wt.value() > 1e-30f)) return -1;
    const float d = (float)decay[n], d4 = 0.25f * d;
    constexpr uint32_t kMagic = 0x4b000000u;
    uint32_t e4 = 4u * (uint32_t)excl - kMagic;
    const uint32_t end4 = e4 + 4u * (uint32_t)words.cnt;
    Acc<float> Wl;
    // the extrema, the next best of each, and the hits (times four) they are at
    float mx = -CUDART_INF_F, mx2 = -CUDART_INF_F, mn = CUDART_INF_F, mn2 = CUDART_INF_F;
    uint32_t pmx = ~0u, pmn = ~0u;
    HitWalk<WPL> hit(bmw, w0, words);
#pragma unroll 2
    while (e4 != end4) {
        const uint32_t r4 = hit.next();
        const float m4 = __fadd_rn(__uint_as_float(r4 - e4), -8388608.f);
        const float md = __fmul_rn(-m4, d4);
        const float before = Wl.scaled_plus(inv, md);
        mn2 = fminf(mn2, fmaxf(mn, before));
        pmn = before < mn ? r4 : pmn;
        mn = fminf(mn, before);
        Wl.add(wf(r4));
        const float after = Wl.scaled_plus(inv, md);
        mx2 = fmaxf(mx2, fminf(mx, after));
        pmx = after > mx ? r4 : pmx;
        mx = fmaxf(mx, after);
        e4 += 4u;
    }
    const float shift = weight_before<float>(Wl, excl, inv, lane);
    mx += shift;
    mx2 += shift;
    mn += shift;
    mn2 += shift;
    if (lane == 31) {  // end of the list: no hit to evaluate at
        const float end = Wt.scaled_plus(inv, -(float)(G - n) * d);
        mn2 = fminf(mn2, fmaxf(mn, end));
        if (end < mn) {
            mn = end;
            pmn = ~0u;
        }
    }
    const float up = __uint_as_float(warp_top(mx)), down = __uint_as_float(warp_top(-mn));
    largest = up > down;
    if (fabsf(up - down) <= kMargin) return -1;
    const float lead = largest ? up : -down;
    const float first = largest ? mx : -mn, second = largest ? mx2 : -mn2;
    const uint32_t near = __ballot_sync(kFullMask, first >= fabsf(lead) - kMargin);
    const bool tied = __any_sync(kFullMask, second >= fabsf(lead) - kMargin);
    if (tied || (near & (near - 1u)) != 0u || near == 0u) return -1;
    const uint32_t at = __shfl_sync(kFullMask, largest ? pmx : pmn, __ffs((int)near) - 1);
    return at == ~0u ? -1 : (int)(at >> 2);
}

// General procedure (any G, any set size): each lane walks its own word range
// twice -- weights first, then candidates with the exact prefix from a scan.
template <class T>
__device__ __noinline__ T set_score_walk(uint32_t* bm, int w0, int w1, const T* wt, const T* __restrict__ decay,
                                         int G, int lane) {
    int h = 0;
    Acc<T> Wl;
    for (int w = w0; w < w1; w++) {
        uint32_t word = bm[w];
        h += __popc(word);
        while (word) {
            const int bit = __ffs(word) - 1;
            word &= word - 1;
            Wl.add(wt[(w << 5) + bit]);
        }
    }
    int h_incl = h;
    Acc<T> W_incl = Wl;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int hy = __shfl_up_sync(kFullMask, h_incl, o);
        const Acc<T> wy = W_incl.shfl_up(o);
        if (lane >= o) {
            h_incl += hy;
            W_incl.merge(wy);
        }
    }
    const int n = __shfl_sync(kFullMask, h_incl, 31);
    Acc<T> Wt;
    Wt.hi = __shfl_sync(kFullMask, W_incl.hi, 31);
    Wt.lo = __shfl_sync(kFullMask, W_incl.lo, 31);
    const T N_R = Wt.value();
    const T inv = n > 0 ? T(1) / N_R : T(0);
    const T d = decay[n];
    Acc<T> W = W_incl.shfl_up(1);
    if (lane == 0) W = Acc<T>();
    int j = h_incl - h;
    T best = T(0);
    int bpos = -1;
    for (int w = w0; w < w1; w++) {
        uint32_t word = bm[w];
        if (!word) continue;
        bm[w] = 0u;
        while (word) {
            const int bit = __ffs(word) - 1;
            word &= word - 1;
            const int r = (w << 5) + bit;
            const T m = (T)(r - j);
            const T before = j > 0 ? W.scaled_plus(inv, -m * d) : -m * d;
            consider<T>(before, r - 1, best, bpos);
            W.add(wt[r]);
            j++;
            consider<T>(W.scaled_plus(inv, -m * d), r, best, bpos);
        }
    }
    if (lane == 31) {
        const T tail = -(T)(G - n) * d;
        consider<T>(n > 0 ? Wt.scaled_plus(inv, tail) : tail, G - 1, best, bpos);
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        const T ob = __shfl_xor_sync(kFullMask, best, o);
        const int op = __shfl_xor_sync(kFullMask, bpos, o);
        consider<T>(ob, op, best, bpos);
    }
    return best;
}

// a member's rank in the direct procedures' bitmap: bit 31 - r % 32
template <int WPL>
__device__ __forceinline__ void mark(uint32_t* bm, uint32_t r) {
    atomicOr(rank_word<WPL>(bm, r), __funnelshift_r(0x80000000u, 0u, r));
}

// One permutation on the calling CTA: stage its ranks and weights (STAGE 1),
// its ranks only (STAGE 2, the weights then gathered through L1 / L2), its
// weights only (STAGE 3, the ranks gathered) or nothing (STAGE 0),
// then warps take sets from the CTA-wide counter until the CTA's share is
// scored.  The share is parts [part_lo, part_hi) of `parts` interleaved parts
// of the set order (part j: slots j, j + parts, j + 2*parts, ...), so that
// every part mixes large and small sets; parts = 1 takes every set.
// s_w / s_rank: staging (STAGE), bm: this warp's zeroed bitmap region.
// Begins and ends with the CTA in step (the staging may be reused after).
template <class T, class RankT, int WARPS, int STAGE, int WPL>
__device__ __forceinline__ void es_one_perm(const RankT* rk, const T* wt, int G, const EsSets sets,
                                            const int32_t* __restrict__ set_order, const T* __restrict__ decay, int K,
                                            T* __restrict__ es_col, int64_t es_stride, T* s_w, RankT* s_rank,
                                            uint32_t* bm, int* next_set, int part_lo = 0, int part_hi = 1,
                                            int parts = 1) {
    // the general procedure reads weights of type T; 16-bit ranks have room
    // for floats only (es_weight_bytes)
    static_assert(WPL > 0 || sizeof(RankT) == 4, "16-bit ranks take the direct procedures");
    const int tid = threadIdx.x, lane = tid & 31;
    const int words = (G + 31) >> 5;
    const int wpl = WPL > 0 ? WPL : (words + 31) >> 5;  // bitmap words per lane
    const int w0 = min(lane * wpl, words), w1 = min(w0 + wpl, words);
    __syncthreads();  // previous permutation finished with the staging and the counter
    if (tid == 0) *next_set = 0;
    constexpr bool F64 = std::is_same<T, double>::value && WPL > 0;  // walk in fp32, score from double sums
    float* const s_wf = reinterpret_cast<float*>(s_w);
    if (STAGE) {
        for (int i = tid; i < G; i += WARPS * 32) {
            if (STAGE == 1 || STAGE == 3) {
                if constexpr (F64) s_wf[i] = (float)wt[i];
                else s_w[i] = wt[i];
            }
            if (STAGE == 1 || STAGE == 2) s_rank[i] = rk[i];
        }
        if (STAGE == 1 || STAGE == 2) rk = s_rank;
        if ((STAGE == 1 || STAGE == 3) && !F64) wt = s_w;
    }
    // fp64: the scores of up to 32 sets wait in the lanes for their division
    double up_to = 0.0, beyond = 0.0;  // weight up to the extremum, weight after it
    int misses = 0, hits = 0, waiting = -1, held = 0;
    auto flush = [&]() {
        if constexpr (F64) {
            if (waiting >= 0) {
                const double inv = 1.0 / (up_to + beyond);
                es_col[(int64_t)waiting * es_stride] = fma(up_to, inv, -(double)misses * decay[hits]);
            }
            waiting = -1;
            held = 0;
        }
    };
    __syncthreads();
    while (true) {
        int slot = 0;
        if (lane == 0) slot = atomicAdd(next_set, 1);
        slot = __shfl_sync(kFullMask, slot, 0);
        if (parts > 1) {  // i-th set of the share: slots grow with i
            const int m = part_hi - part_lo;
            slot = (slot / m) * parts + part_lo + slot % m;
        }
        if (slot >= K) break;
        const int k = set_order ? set_order[slot] : slot;
        T score;
        if constexpr (WPL > 0) {
            auto weight = [&](uint32_t r) -> float {
                if constexpr (F64) return STAGE == 1 || STAGE == 3 ? s_wf[r] : (float)wt[r];
                else return wt[r];
            };
            Acc<float> Wm;
            const int2 rec = __ldg(sets.rec + k);  // first group of the set's list, members
            const uint2* __restrict__ const list = sets.list + (int64_t)(rec.x < 0 ? ~rec.x : rec.x) * 32 + lane;
            const int full = rec.y >> 7, rem = rec.y & 127;
            if (F64 || rec.x >= 0) {
#pragma unroll 1
                for (int i = 0; i < full; i++) {
                    const uint2 q = __ldg(list + 32 * i);
                    const uint32_t r0 = rk[q.x & 0xffffu], r1 = rk[q.x >> 16];
                    const uint32_t r2 = rk[q.y & 0xffffu], r3 = rk[q.y >> 16];
                    const float a0 = weight(r0), a1 = weight(r1), a2 = weight(r2), a3 = weight(r3);
                    mark<WPL>(bm, r0);
                    mark<WPL>(bm, r1);
                    mark<WPL>(bm, r2);
                    mark<WPL>(bm, r3);
                    Wm.add(a0);
                    Wm.add(a1);
                    Wm.add(a2);
                    Wm.add(a3);
                }
                if (rem) {
                    const uint2 q = __ldg(list + 32 * full);
                    const uint32_t g[4] = {q.x & 0xffffu, q.x >> 16, q.y & 0xffffu, q.y >> 16};
                    uint32_t r[4];
                    float a[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) {  // the unused entries of a list are gene 0
                        r[i] = rk[g[i]];
                        a[i] = weight(r[i]);
                    }
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        if (lane + 32 * i < rem) {
                            mark<WPL>(bm, r[i]);
                            Wm.add(a[i]);
                        }
                    }
                }
            } else {
                // duplicates or unknown ids: the caller's list, each member checked
                const int64_t a = sets.off[k];
                const int m = (int)(sets.off[k + 1] - a);  // a set lists fewer than 2^31 members
                for (int64_t base = 0; base < m; base += 128) {
                    int g[4];
                    uint32_t r[4];
                    float w[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const int64_t idx = base + lane + 32 * i;
                        g[i] = idx < m ? __ldg(sets.genes + a + idx) : -1;
                    }
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        r[i] = rk[g[i] >= 0 && g[i] < G ? g[i] : 0];
                        w[i] = weight(r[i]);
                    }
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        if (g[i] >= 0 && g[i] < G) {
                            const uint32_t bit = __funnelshift_r(0x80000000u, 0u, r[i]);
                            if (!(atomicOr(rank_word<WPL>(bm, r[i]), bit) & bit)) Wm.add(w[i]);
                        }
                    }
                }
            }
            __syncwarp();
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) Wm.merge(Wm.shfl_xor(o));  // the set's weight, every lane
            uint32_t* const bmw = bm + lane * lane_stride<WPL>();
            if constexpr (!F64) {
                score = set_score_direct<WPL>(bmw, lane * WPL, wt, decay, G, lane, Wm);
                clear_words<WPL>(bmw);
            } else {
                int n;
                bool largest;
                const int at = find_extremum<WPL>(
                    bmw, lane * WPL,
                    [&](uint32_t r4) -> float {
                        if constexpr (STAGE == 1 || STAGE == 3) return weight_at(s_wf, r4);
                        else return (float)weight_at(wt, r4);
                    },
                    decay, G, lane, Wm, n, largest);
                if (at < 0) {  // warp-uniform
                    score = set_score_positions_f64<WPL>(bmw, lane * WPL, wt, rk, list, rec.y, decay, G, lane);
                    clear_words<WPL>(bmw);
                } else {
                    clear_words<WPL>(bmw);
                    // the members' weights once more, in double, on either side
                    // of the extremum: one addition a member
                    const uint32_t limit = (uint32_t)at + (largest ? 1u : 0u);
                    double lo = 0.0, hi = 0.0;
                    int before = 0;
                    auto add = [&](uint32_t r, double w) {
                        const bool in = r < limit;
                        const double sum = (in ? lo : hi) + w;
                        lo = in ? sum : lo;
                        hi = in ? hi : sum;
                        before += r < (uint32_t)at ? 1 : 0;
                    };
#pragma unroll 1
                    for (int i = 0; i < full; i++) {
                        const uint2 q = __ldg(list + 32 * i);
                        const uint32_t r0 = rk[q.x & 0xffffu], r1 = rk[q.x >> 16];
                        const uint32_t r2 = rk[q.y & 0xffffu], r3 = rk[q.y >> 16];
                        const double a0 = wt[r0], a1 = wt[r1], a2 = wt[r2], a3 = wt[r3];
                        add(r0, a0);
                        add(r1, a1);
                        add(r2, a2);
                        add(r3, a3);
                    }
                    if (rem) {
                        const uint2 q = __ldg(list + 32 * full);
                        const uint32_t g[4] = {q.x & 0xffffu, q.x >> 16, q.y & 0xffffu, q.y >> 16};
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            if (lane + 32 * i < rem) {
                                const uint32_t r = rk[g[i]];
                                add(r, wt[r]);
                            }
                        }
                    }
                    before = __reduce_add_sync(kFullMask, before);
                    // both sums in five steps: after the first, lanes 0-15 hold
                    // one and lanes 16-31 the other
                    double mine = (lane < 16 ? lo : hi) + __shfl_xor_sync(kFullMask, lane < 16 ? hi : lo, 16);
#pragma unroll
                    for (int o = 8; o >= 1; o >>= 1) mine += __shfl_xor_sync(kFullMask, mine, o);
                    const double s_lo = __shfl_sync(kFullMask, mine, 0), s_hi = __shfl_sync(kFullMask, mine, 16);
                    if (lane == held) {
                        up_to = s_lo;
                        beyond = s_hi;
                        misses = at - before;
                        hits = n;
                        waiting = k;
                    }
                    if (++held == 32) flush();
                    __syncwarp();
                    continue;
                }
            }
        } else {
            // mark the members' ranks (duplicates and unknown ids fall away)
            const int64_t a = sets.off[k];
            const int m = (int)(sets.off[k + 1] - a);
            for (int idx = lane; idx < m; idx += 32) {
                const int g = __ldg(sets.genes + a + idx);
                if (g >= 0 && g < G) {
                    const uint32_t r = (uint32_t)rk[g];
                    atomicOr(&bm[r >> 5], 1u << (r & 31));
                }
            }
            __syncwarp();
            score = set_score_walk<T>(bm, w0, w1, wt, decay, G, lane);
        }
        if (lane == 0) es_col[(int64_t)k * es_stride] = score;
        __syncwarp();
    }
    flush();
}

// bytes of a CTA's staging: weights + ranks (1), ranks (2), weights (3), none
// (0); the direct procedures stage fp64 weights as floats (the walk's)
template <class T, class RankT>
__host__ __device__ constexpr size_t es_weight_bytes() { return sizeof(RankT) == 2 ? 4 : sizeof(T); }
template <class T, class RankT, int STAGE>
__host__ __device__ __forceinline__ size_t es_stage_bytes(int G) {
    return STAGE == 1   ? (es_weight_bytes<T, RankT>() + sizeof(RankT)) * (size_t)G
           : STAGE == 2 ? sizeof(RankT) * (size_t)G
           : STAGE == 3 ? es_weight_bytes<T, RankT>() * (size_t)G
                        : 0;
}

// shared memory of a CTA: staging for G genes (STAGE) + WARPS bitmap regions
template <class T, class RankT, int STAGE>
__device__ __forceinline__ void es_smem_layout(unsigned char* smem, int G, int region, T*& s_w, RankT*& s_rank,
                                               uint32_t*& bm) {
    const int warp = threadIdx.x >> 5;
    s_w = reinterpret_cast<T*>(smem);
    s_rank = reinterpret_cast<RankT*>(smem + (STAGE == 1 ? es_weight_bytes<T, RankT>() * (size_t)G : 0));
    size_t bm_off = es_stage_bytes<T, RankT, STAGE>(G);
    bm_off = (bm_off + 15) & ~(size_t)15;
    bm = reinterpret_cast<uint32_t*>(smem + bm_off) + (size_t)warp * region;
}

// 16 warps with everything staged come as two CTAs to an SM (launch_es_t)
template <class T, int WARPS, int STAGE>
constexpr bool pairs_up() {
    return sizeof(T) == 4 && WARPS == 16 && STAGE == 1;
}

// WPL > 0: bitmap words per lane held in registers by the list procedure
// (G <= 1024*WPL, 16-bit ranks); WPL == 0: general procedure (32-bit ranks).
template <class T, class RankT, int WARPS, int STAGE, int WPL>
__global__ void __launch_bounds__(WARPS * 32, pairs_up<T, WARPS, STAGE>() ? 2 : 1)
es_kernel(const RankT* __restrict__ ranks, const T* __restrict__ sorted_abs, int G, int num_perms,
          const EsSets sets, const int32_t* __restrict__ set_order, const T* __restrict__ decay, int K,
          T* __restrict__ es, int64_t es_stride, int64_t col0, const int* __restrict__ K_dev) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int next_set;
    if (K_dev) K = min(K, *K_dev);  // a set list whose length a kernel decided
    if (K <= 0) return;
    const int words = (G + 31) >> 5;
    const int region = WPL > 0 ? lane_stride<WPL>() * 32 : words;  // per-warp bitmap words
    T* s_w;
    RankT* s_rank;
    uint32_t* bm;
    es_smem_layout<T, RankT, STAGE>(smem, G, region, s_w, s_rank, bm);
    for (int w = threadIdx.x & 31; w < region; w += 32) bm[w] = 0u;
    // whole permutations in rounds of gridDim.x ...
    const int grid = gridDim.x;
    const int full = num_perms / grid;
    for (int i = 0; i < full; i++) {
        const int p = blockIdx.x + i * grid;
        es_one_perm<T, RankT, WARPS, STAGE, WPL>(ranks + (int64_t)p * G, sorted_abs + (int64_t)p * G, G, sets,
                                                  set_order, decay, K, es + col0 + p, es_stride, s_w, s_rank, bm,
                                                  &next_set);
    }
    // ... then the rem < gridDim.x left over, each cut into `parts` parts
    // (parts * rem a multiple of gridDim.x where K allows); every CTA takes an
    // equal contiguous run of the (permutation, part) items, which spans at
    // most a few permutations, so the last round ends evenly
    const int rem = num_perms - full * grid;
    if (rem == 0) return;
    int a = rem, b = grid;
    while (b) { const int t = a % b; a = b; b = t; }
    const int parts = min(grid / a, K);
    const int64_t items = (int64_t)rem * parts;
    int64_t lo = items * blockIdx.x / grid;
    const int64_t hi = items * (blockIdx.x + 1) / grid;
    while (lo < hi) {
        const int64_t q = lo / parts;
        const int j0 = (int)(lo - q * parts);
        const int64_t left = hi - lo;
        const int j1 = left < (int64_t)(parts - j0) ? j0 + (int)left : parts;
        const int p = full * grid + (int)q;
        es_one_perm<T, RankT, WARPS, STAGE, WPL>(ranks + (int64_t)p * G, sorted_abs + (int64_t)p * G, G, sets,
                                                  set_order, decay, K, es + col0 + p, es_stride, s_w, s_rank, bm,
                                                  &next_set, j0, j1, parts);
        lo += j1 - j0;
    }
}

// Persistent multi-instance form: every CTA takes (instance, permutation)
// items from a global counter until all are done; items run in task order
// (tasks sorted by decreasing cost by the caller) and a task's permutations
// in order.  item_end[t] = items of tasks 0..t; Gmax sizes the staging and
// the bitmap regions of the size class (every task: G <= Gmax <= 1024*WPL).
template <class T, class RankT, int WARPS, int STAGE, int WPL>
__global__ void __launch_bounds__(WARPS * 32)
es_batch_kernel(const EsTask<T>* __restrict__ tasks, const int64_t* __restrict__ item_end, int ntasks,
                int64_t nitems, unsigned long long* __restrict__ counter, int Gmax) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int next_set;
    __shared__ long long s_item;
    const int region = lane_stride<WPL>() * 32;
    T* s_w;
    RankT* s_rank;
    uint32_t* bm;
    es_smem_layout<T, RankT, STAGE>(smem, Gmax, region, s_w, s_rank, bm);
    for (int w = threadIdx.x & 31; w < region; w += 32) bm[w] = 0u;
    while (true) {
        __syncthreads();  // everyone read s_item of the previous round
        if (threadIdx.x == 0) s_item = (long long)atomicAdd(counter, 1ull);
        __syncthreads();
        const int64_t item = s_item;
        if (item >= nitems) break;
        int lo = 0, hi = ntasks - 1;  // first task with item_end > item
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (item_end[mid] > item) hi = mid; else lo = mid + 1;
        }
        const EsTask<T>& tk = tasks[lo];
        const int64_t p = item - (lo > 0 ? item_end[lo - 1] : 0);
        const RankT* rk = static_cast<const RankT*>(tk.ranks) + p * tk.G;
        es_one_perm<T, RankT, WARPS, STAGE, WPL>(rk, tk.sorted + p * tk.G, tk.G, tk.sets, tk.order, tk.decay, tk.K,
                                                  tk.es + tk.col0 + p, tk.stride, s_w, s_rank, bm, &next_set);
    }
}

// words of a warp's bitmap region
inline int es_region_words(int G, int wpl) {
    return wpl > 0 ? (wpl % 16 == 0 ? wpl + 4 : wpl) * 32 : (G + 31) >> 5;
}

inline int es_wpl(int G, bool ranks16) {
    const int need = (((G + 31) >> 5) + 31) >> 5;
    if (!ranks16) return 0;
    for (int w : {4, 8, 12, 16, 20, 24, 32, 40, 48, 64})
        if (need <= w) return w;
    return 0;
}

template <class T, class RankT, int WARPS, int STAGE>
size_t es_smem_bytes(int G) {
    const int region = es_region_words(G, es_wpl(G, sizeof(RankT) == 2));
    const size_t s = (es_stage_bytes<T, RankT, STAGE>(G) + 15) & ~(size_t)15;
    return s + sizeof(uint32_t) * (size_t)region * WARPS;
}

// Whether a configuration may run.  The first pass over the candidates leaves
// an unstaged one at least 64 KB of the SM's memory as L1: its gathers of
// ranks and weights live there (60,000 genes, 304 x 500 scores: 24 warps
// with 28 KB of L1 772 us, 16 warps with 92 KB 477; 45,000: 32 warps 731, 24
// warps 380), so more warps are only worth it while the bitmaps stay below
// 164 KB.
// `asked`: what an explicit request of staged weights must leave room for
// (fp64: the weights themselves, though the kernel stages them as floats).
inline bool es_fits(int warps, int stage, size_t smem, size_t asked, int wpl, size_t cap, bool leave_l1,
                    const EsTuning& tune) {
    constexpr size_t kLeavesL1 = 163 * 1024;
    if (smem + (tune.stage == 1 || tune.stage == 3 ? asked : 0) > cap) return false;
    if ((stage >= 2 || warps == 24) && wpl < 24) return false;
    if (stage == 1 && wpl >= 40) return false;
    if (tune.warps && tune.warps != warps) return false;
    if (tune.stage >= 0 && tune.stage != stage) return false;
    return !(leave_l1 && stage == 0 && smem > kLeavesL1);
}

// Launch with the shared memory of the resident CTAs and all the L1 that
// leaves: what is not staged is gathered through L1.  Without the request an
// SM keeps the split of the kernel that ran on it before, the sort's with
// hardly any L1, whenever passes on several streams leave it no idle moment
// (passes of several plans in turn: 60,000 genes 1,183 -> 948 us, 36,161 genes
// 1,554 -> 1,145; a single plan's the same, all staged the same; all of it as
// shared memory 1,219 and 1,636).
template <class... P, class... A>
cudaError_t launch_es_kernel(void (*kern)(P...), int grid, int warps, size_t smem, int per_sm, cudaStream_t st,
                             A... args) {
    int dev = 0, all = 0, reserved = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&all, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
    cudaLaunchAttribute l1;
    l1.id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    // per cent, rounded down: the split in use is the next larger one
    l1.val.sharedMemCarveout =
        (unsigned)std::min<size_t>(100, (size_t)per_sm * (smem + (size_t)reserved) * 100 / (size_t)std::max(all, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)warps * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &l1;
    cfg.numAttrs = 1;
    launches_add(1);
    return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

template <class T, class RankT, int WARPS, int STAGE, int WPL>
cudaError_t launch_es_v(const RankT* ranks, const T* sorted_abs, int G, int P, const EsSets& sets,
                        const int32_t* order, const T* decay, int K, T* es, int64_t stride,
                        int64_t col0, int grid, cudaStream_t st, const int* K_dev) {
    const size_t smem = es_smem_bytes<T, RankT, WARPS, STAGE>(G);
    auto kern = es_kernel<T, RankT, WARPS, STAGE, WPL>;
    cudaError_t e = allow_smem(kern, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;  // resident CTAs per SM: the grid fills the device once
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, WARPS * 32, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidValue;
    return launch_es_kernel(kern, grid * per_sm, WARPS, smem, per_sm, st, ranks, sorted_abs, G, P, sets, order, decay,
                            K, es, stride, col0, K_dev);
}

template <class T, class RankT, int WARPS, int STAGE>
cudaError_t launch_es_w(const RankT* ranks, const T* sorted_abs, int G, int P, const EsSets& sets,
                        const int32_t* order, const T* decay, int K, T* es, int64_t stride,
                        int64_t col0, int grid, cudaStream_t st, const int* K_dev) {
    // words per lane for the register-resident list procedure (u16 positions);
    // 32-bit ranks (G > 65,536) always take the general procedure
    if constexpr (sizeof(RankT) == 4) {
        if (STAGE >= 2) return cudaErrorInvalidValue;
        return launch_es_v<T, RankT, WARPS, STAGE, 0>(ranks, sorted_abs, G, P, sets, order, decay, K, es, stride,
                                                      col0, grid, st, K_dev);
    } else if constexpr (STAGE >= 2 || WARPS == 24) {  // partial staging / 24 warps: the large-G classes
        switch (es_wpl(G, true)) {
            case 24: return launch_es_v<T, RankT, WARPS, STAGE, 24>(ranks, sorted_abs, G, P, sets, order, decay, K, es, stride, col0, grid, st, K_dev);
            case 32: return launch_es_v<T, RankT, WARPS, STAGE, 32>(ranks, sorted_abs, G, P, sets, order, decay, K, es, stride, col0, grid, st, K_dev);
            case 40: return launch_es_v<T, RankT, WARPS, STAGE, 40>(ranks, sorted_abs, G, P, sets, order, decay, K, es, stride, col0, grid, st, K_dev);
            case 48: return launch_es_v<T, RankT, WARPS, STAGE, 48>(ranks, sorted_abs, G, P, sets, order, decay, K, es, stride, col0, grid, st, K_dev);
            case 64: return launch_es_v<T, RankT, WARPS, STAGE, 64>(ranks, sorted_abs, G, P, sets, order, decay, K, es, stride, col0, grid, st, K_dev);
            default: return cudaErrorInvalidValue;
        }
    } else {
        switch (es_wpl(G, true)) {
            case 4: return launch_es_v<T, RankT, WARPS, STAGE, 4>(ranks, sorted_abs, G, P, sets, order, decay, K, es, stride, col0, grid, st, K_dev);
            case 8: return launch_es_v<T, RankT, WARPS, STAGE, 8>(ranks, sorted_abs, G, P, sets, order, decay, K, es, stride, col0, grid, st, K_dev);
            case 12: return launch_es_v<T, RankT, WARPS, STAGE, 12>(ranks, sorted_abs, G, P, sets, order, decay, K, es, stride, col0, grid, st, K_dev);
            case 16: return launch_es_v<T, RankT, WARPS, STAGE, 16>(ranks, sorted_abs, G, P, sets, order, decay, K, es, stride, col0, grid, st, K_dev);
            case 20: return launch_es_v<T, RankT, WARPS, STAGE, 20>(ranks, sorted_abs, G, P, sets, order, decay, K, es, stride, col0, grid, st, K_dev);
            case 24: return launch_es_v<T, RankT, WARPS, STAGE, 24>(ranks, sorted_abs, G, P, sets, order, decay, K, es, stride, col0, grid, st, K_dev);
            case 32: return launch_es_v<T, RankT, WARPS, STAGE, 32>(ranks, sorted_abs, G, P, sets, order, decay, K, es, stride, col0, grid, st, K_dev);
            case 40:  // the staging of ranks and weights never fits beside these regions
                if constexpr (STAGE == 0) return launch_es_v<T, RankT, WARPS, 0, 40>(ranks, sorted_abs, G, P, sets, order, decay, K, es, stride, col0, grid, st, K_dev);
                return cudaErrorInvalidValue;
            case 48:
                if constexpr (STAGE == 0) return launch_es_v<T, RankT, WARPS, 0, 48>(ranks, sorted_abs, G, P, sets, order, decay, K, es, stride, col0, grid, st, K_dev);
                return cudaErrorInvalidValue;
            case 64:
                if constexpr (STAGE == 0) return launch_es_v<T, RankT, WARPS, 0, 64>(ranks, sorted_abs, G, P, sets, order, decay, K, es, stride, col0, grid, st, K_dev);
                return cudaErrorInvalidValue;
            default: return cudaErrorInvalidValue;  // none: es_wpl covers every G of 16-bit ranks
        }
    }
}

template <class T, class RankT>
cudaError_t launch_es_t(const RankT* ranks, const T* sorted_abs, int G, int P, const EsSets& sets,
                        const int32_t* order, const T* decay, int K, T* es, int64_t stride,
                        int64_t col0, EsTuning tune, cudaStream_t st, const int* K_dev) {
    int dev = 0, max_smem = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const size_t cap = (size_t)max_smem - 64;  // static shared counter
    const int grid = sms;  // times the resident CTAs per SM; the last round's permutations are split by sets
    // candidates in the automatic order (es_fits): staging the weights first,
    // 32 warps, then 24; then the ranks at 24 warps (36,161 genes, 116 x 4,105
    // scores: 1,049 us, against 1,102 for 32 warps and nothing staged); then
    // nothing.  The partial stagings are for the large-G classes (24-64 bitmap
    // words per lane)
    struct Cand { int warps; int stage; size_t smem; };
    const Cand cands[] = {{32, 1, es_smem_bytes<T, RankT, 32, 1>(G)},
                          {32, 3, es_smem_bytes<T, RankT, 32, 3>(G)},
                          {24, 3, es_smem_bytes<T, RankT, 24, 3>(G)},
                          {24, 2, es_smem_bytes<T, RankT, 24, 2>(G)},
                          {32, 0, es_smem_bytes<T, RankT, 32, 0>(G)},
                          {24, 0, es_smem_bytes<T, RankT, 24, 0>(G)},
                          {16, 0, es_smem_bytes<T, RankT, 16, 0>(G)},
                          {32, 2, es_smem_bytes<T, RankT, 32, 2>(G)},
                          {16, 1, es_smem_bytes<T, RankT, 16, 1>(G)},
                          {16, 2, es_smem_bytes<T, RankT, 16, 2>(G)},
                          {8, 1, es_smem_bytes<T, RankT, 8, 1>(G)},
                          {8, 0, es_smem_bytes<T, RankT, 8, 0>(G)}};
    const int wpl = es_wpl(G, sizeof(RankT) == 2);
#define GSEA_ES(W, S) \
    return launch_es_w<T, RankT, W, S>(ranks, sorted_abs, G, P, sets, order, decay, K, es, stride, col0, grid, st, \
                                       K_dev)
    // Few sets to a permutation: two CTAs of 16 warps, of which one scores while
    // the other stages its permutation or waits for its last sets.  50 sets x
    // 1,024 permutations, 2,000 genes: 86 -> 82 us (passes in turn 128 -> 119),
    // 12,000 genes 88 -> 82; 250 sets 287 -> 281, 300 sets 373 -> 373, 600 sets
    // 367 -> 379.  With fewer permutations than SMs both halves stage the same
    // ones (200 sets, 1,000 genes, 130 permutations 57 us with 32 warps, 69 with
    // pairs; 12,000 genes 41 and 49; 152 permutations 57 and 59, 39 and 41): only
    // where the sets are so few that the smaller CTAs, which run beside another
    // pass's kernels, matter more (66 sets x 272, 3,551 genes, passes of several
    // plans in turn: 52 us with 32 warps, 46 with pairs).
    if constexpr (pairs_up<T, 16, 1>()) {
        int all = 0, reserved = 0;
        cudaDeviceGetAttribute(&all, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
        cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
        const size_t pair = 2 * (es_smem_bytes<T, RankT, 16, 1>(G) + 64 + (size_t)reserved);
        if ((K <= 64 || (K <= 256 && P >= sms)) && !tune.warps && tune.stage < 0 && wpl < 40 && pair <= (size_t)all) GSEA_ES(16, 1);
    }
    for (int pass = 0; pass < 2; pass++)
    for (const Cand& c : cands) {
        if (!es_fits(c.warps, c.stage, c.smem, (sizeof(T) - es_weight_bytes<T, RankT>()) * (size_t)G, wpl, cap,
                     pass == 0, tune))
            continue;
        if (c.warps == 32 && c.stage == 1) GSEA_ES(32, 1);
        if (c.warps == 16 && c.stage == 1) GSEA_ES(16, 1);
        if (c.warps == 8 && c.stage == 1) GSEA_ES(8, 1);
        if (c.warps == 32 && c.stage == 3) GSEA_ES(32, 3);
        if (c.warps == 24 && c.stage == 3) GSEA_ES(24, 3);
        if (c.warps == 32 && c.stage == 2) GSEA_ES(32, 2);
        if (c.warps == 24 && c.stage == 2) GSEA_ES(24, 2);
        if (c.warps == 24 && c.stage == 0) GSEA_ES(24, 0);
        if (c.warps == 16 && c.stage == 2) GSEA_ES(16, 2);
        if (c.warps == 32) GSEA_ES(32, 0);
        if (c.warps == 16) GSEA_ES(16, 0);
        GSEA_ES(8, 0);
#undef GSEA_ES
    }
    return cudaErrorInvalidValue;  // the requested configuration does not fit
}

template <class T, int WARPS, int STAGE, int WPL>
cudaError_t launch_es_batch_v(const EsTask<T>* tasks, const int64_t* item_end, int ntasks, int64_t nitems,
                              unsigned long long* counter, int Gmax, cudaStream_t st) {
    const size_t smem = es_smem_bytes<T, uint16_t, WARPS, STAGE>(Gmax);
    auto kern = es_batch_kernel<T, uint16_t, WARPS, STAGE, WPL>;
    cudaError_t e = allow_smem(kern, smem);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 1, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, WARPS * 32, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidValue;
    const int64_t want = (int64_t)sms * per_sm;
    const int grid = (int)(nitems < want ? nitems : want);
    e = cudaMemsetAsync(counter, 0, sizeof(unsigned long long), st);
    if (e != cudaSuccess) return e;
    return launch_es_kernel(kern, grid, WARPS, smem, per_sm, st, tasks, item_end, ntasks, nitems, counter, Gmax);
}

template <class T, int WARPS, int STAGE>
cudaError_t launch_es_batch_w(const EsTask<T>* tasks, const int64_t* item_end, int ntasks, int64_t nitems,
                              unsigned long long* counter, int Gmax, int wpl, cudaStream_t st) {
    if constexpr (STAGE >= 2 || WARPS == 24) {
        switch (wpl) {
            case 24: return launch_es_batch_v<T, WARPS, STAGE, 24>(tasks, item_end, ntasks, nitems, counter, Gmax, st);
            case 32: return launch_es_batch_v<T, WARPS, STAGE, 32>(tasks, item_end, ntasks, nitems, counter, Gmax, st);
            case 40: return launch_es_batch_v<T, WARPS, STAGE, 40>(tasks, item_end, ntasks, nitems, counter, Gmax, st);
            case 48: return launch_es_batch_v<T, WARPS, STAGE, 48>(tasks, item_end, ntasks, nitems, counter, Gmax, st);
            case 64: return launch_es_batch_v<T, WARPS, STAGE, 64>(tasks, item_end, ntasks, nitems, counter, Gmax, st);
            default: return cudaErrorInvalidValue;
        }
    } else {
    switch (wpl) {
        case 4: return launch_es_batch_v<T, WARPS, STAGE, 4>(tasks, item_end, ntasks, nitems, counter, Gmax, st);
        case 8: return launch_es_batch_v<T, WARPS, STAGE, 8>(tasks, item_end, ntasks, nitems, counter, Gmax, st);
        case 12: return launch_es_batch_v<T, WARPS, STAGE, 12>(tasks, item_end, ntasks, nitems, counter, Gmax, st);
        case 16: return launch_es_batch_v<T, WARPS, STAGE, 16>(tasks, item_end, ntasks, nitems, counter, Gmax, st);
        case 20: return launch_es_batch_v<T, WARPS, STAGE, 20>(tasks, item_end, ntasks, nitems, counter, Gmax, st);
        case 24: return launch_es_batch_v<T, WARPS, STAGE, 24>(tasks, item_end, ntasks, nitems, counter, Gmax, st);
        case 32: return launch_es_batch_v<T, WARPS, STAGE, 32>(tasks, item_end, ntasks, nitems, counter, Gmax, st);
        case 40:
            if constexpr (STAGE == 0) return launch_es_batch_v<T, WARPS, 0, 40>(tasks, item_end, ntasks, nitems, counter, Gmax, st);
            return cudaErrorInvalidValue;
        case 48:
            if constexpr (STAGE == 0) return launch_es_batch_v<T, WARPS, 0, 48>(tasks, item_end, ntasks, nitems, counter, Gmax, st);
            return cudaErrorInvalidValue;
        case 64:
            if constexpr (STAGE == 0) return launch_es_batch_v<T, WARPS, 0, 64>(tasks, item_end, ntasks, nitems, counter, Gmax, st);
            return cudaErrorInvalidValue;
        default: return cudaErrorInvalidValue;
    }
    }
}

}  // namespace

template <class T>
cudaError_t launch_es_batch(const EsTask<T>* tasks, const int64_t* item_end, int ntasks, int64_t nitems,
                            unsigned long long* counter, int Gmax, int wpl, EsTuning tune, cudaStream_t st) {
    if (nitems <= 0 || ntasks <= 0) return cudaSuccess;
    if (Gmax > 65536 || es_wpl(Gmax, true) != wpl) return cudaErrorInvalidValue;
    int dev = 0, max_smem = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    const size_t cap = (size_t)max_smem - 64;
    struct Cand { int warps; int stage; size_t smem; };
    const Cand cands[] = {{32, 1, es_smem_bytes<T, uint16_t, 32, 1>(Gmax)},
                          {32, 3, es_smem_bytes<T, uint16_t, 32, 3>(Gmax)},
                          {24, 3, es_smem_bytes<T, uint16_t, 24, 3>(Gmax)},
                          {24, 2, es_smem_bytes<T, uint16_t, 24, 2>(Gmax)},
                          {32, 0, es_smem_bytes<T, uint16_t, 32, 0>(Gmax)},
                          {24, 0, es_smem_bytes<T, uint16_t, 24, 0>(Gmax)},
                          {16, 0, es_smem_bytes<T, uint16_t, 16, 0>(Gmax)},
                          {32, 2, es_smem_bytes<T, uint16_t, 32, 2>(Gmax)},
                          {16, 1, es_smem_bytes<T, uint16_t, 16, 1>(Gmax)},
                          {16, 2, es_smem_bytes<T, uint16_t, 16, 2>(Gmax)},
                          {8, 1, es_smem_bytes<T, uint16_t, 8, 1>(Gmax)},
                          {8, 0, es_smem_bytes<T, uint16_t, 8, 0>(Gmax)}};
    for (int pass = 0; pass < 2; pass++)
    for (const Cand& c : cands) {
        if (!es_fits(c.warps, c.stage, c.smem, (sizeof(T) - es_weight_bytes<T, uint16_t>()) * (size_t)Gmax, wpl, cap,
                     pass == 0, tune))
            continue;
#define GSEA_ESB(W, S) return launch_es_batch_w<T, W, S>(tasks, item_end, ntasks, nitems, counter, Gmax, wpl, st)
        if (c.warps == 32 && c.stage == 1) GSEA_ESB(32, 1);
        if (c.warps == 16 && c.stage == 1) GSEA_ESB(16, 1);
        if (c.warps == 8 && c.stage == 1) GSEA_ESB(8, 1);
        if (c.warps == 32 && c.stage == 3) GSEA_ESB(32, 3);
        if (c.warps == 24 && c.stage == 3) GSEA_ESB(24, 3);
        if (c.warps == 32 && c.stage == 2) GSEA_ESB(32, 2);
        if (c.warps == 24 && c.stage == 2) GSEA_ESB(24, 2);
        if (c.warps == 24 && c.stage == 0) GSEA_ESB(24, 0);
        if (c.warps == 16 && c.stage == 2) GSEA_ESB(16, 2);
        if (c.warps == 32) GSEA_ESB(32, 0);
        if (c.warps == 16) GSEA_ESB(16, 0);
        GSEA_ESB(8, 0);
#undef GSEA_ESB
    }
    return cudaErrorInvalidValue;
}

template <class T>
cudaError_t launch_es(const void* ranks, bool ranks16, const T* sorted_abs, int G, int num_perms,
                      const EsSets& sets, const int32_t* set_order, const T* decay, int K, T* es, int64_t es_stride, int64_t perm_col0, cudaStream_t st,
                      EsTuning tune, const int* K_dev) {
    if (num_perms <= 0 || K <= 0) return cudaSuccess;
    if (ranks16)
        return launch_es_t<T, uint16_t>(static_cast<const uint16_t*>(ranks), sorted_abs, G, num_perms, sets,
                                        set_order, decay, K, es, es_stride, perm_col0, tune, st, K_dev);
    return launch_es_t<T, uint32_t>(static_cast<const uint32_t*>(ranks), sorted_abs, G, num_perms, sets,
                                    set_order, decay, K, es, es_stride, perm_col0, tune, st, K_dev);
}

// decay[n] = (T)(1.0 / (G - n)) for n < G, 0 for n = G: the miss step of a
// set with n hits, rounded from double as the reference does
// (enrichment_scores.cuh:178)
template <class T>
__global__ void decay_table_kernel(int G, T* decay) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n <= G) decay[n] = n < G ? (T)(1.0 / (double)(G - n)) : T(0);
}

template <class T>
cudaError_t launch_decay_table(int G, T* decay, cudaStream_t st) {
    decay_table_kernel<T><<<(G + 256) / 256, 256, 0, st>>>(G, decay);
    launches_add(1);
    return cudaGetLastError();
}


}  // namespace gsea
