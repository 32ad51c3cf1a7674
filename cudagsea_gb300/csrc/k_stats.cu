// k_stats.cu -- NES, nominal p, FWER and FDR on the device.
//
// final_statistics (src/include/statistics.cuh:46-117) runs on the host in
// the reference, in the enrichment precision T.  The same arithmetic runs here
// on the GPU:
//   ES_k    = S[k][0]
//   fac_k   = (T)P / sum_p |S[k][p]|        (sequential sum over p, in T,
//                                            statistics.cuh:60-70)
//   NES_k   = ES_k * fac_k
//   NP_k    = #{p : |S[k][p]| >= |ES_k|} / P          (statistics.cuh:72-77)
//   max_p   = max_k S[k][p]*fac_k, min_p likewise     (statistics.cuh:84-97)
//   FWER_k  = #{p : max_p >= NES_k} / P  if NES_k > 0,
//             #{p : min_p <= NES_k} / P  otherwise    (statistics.cuh:99-110)
// so the results are bit-identical to the reference's for identical ES.
//
// FDR (statistics.cuh:112-114 leaves NaN): q-value of the normalised score
// against the null of permutations 1..P-1 of all sets, per sign side:
//   NES* > 0: q = [#{null >= NES*} / #{null >= 0}] / [#{obs >= NES*} / #{obs >= 0}]
//   NES* <= 0: mirrored with <=, capped at 1.
//
// Ragged form (adaptive permutation allocation): set k holds n_k scores in
// row k of a matrix with row stride ld.  fac, NES and NP use the set's own
// n_k columns; FWER uses the first p_fwer columns (those every set has);
// in the FDR null every set carries the same total weight, each of its
// n_k - 1 null scores counting (ld - 1) / (n_k - 1).  With n_k = ld for all
// sets the weights are exactly 1 and the ragged form is the dense one.
#include <algorithm>
#include "common.cuh"
#include "kernels.h"

namespace gsea {
namespace {

struct StatsScratch {
    // fac[K] mx[P] mn[P] (T) | cnt_obs[K] lcount[K] (u64) | sorted_pos[K]
    // sorted_neg[K] (T) | hpos[K+2] hneg[K+2] (f64) | totals[8] (u64 / f64)
    static size_t bytes(int K, int64_t P, size_t tsize) {
        return tsize * ((size_t)3 * K + 2 * (size_t)P) + sizeof(unsigned long long) * (4 * (size_t)K + 12) + 64;
    }
};

// one warp per set: factor, NES, NP
template <class T>
__device__ __forceinline__ void stats_set_kernel_body(int bx, const T* __restrict__ es, int K, int64_t ld, const int64_t* __restrict__ counts,
                                 T* __restrict__ out, T* __restrict__ fac) {
    const int warp = (bx * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= K) return;
    const T* row = es + (int64_t)warp * ld;
    const int64_t P = counts ? counts[warp] : ld;
    const T es0 = row[0];
    T sum = T(0);
    unsigned long long np = 0;
    const T aes0 = fabs(es0);
    // blocks of 4 x 32 columns; the next block's loads are in flight while
    // this block is summed
    constexpr int kB = 4;
    T cur[kB];
#pragma unroll
    for (int j = 0; j < kB; j++) cur[j] = j * 32 + lane < P ? row[j * 32 + lane] : T(0);
    for (int64_t p0 = 0; p0 < P; p0 += kB * 32) {
        T nxt[kB];
#pragma unroll
        for (int j = 0; j < kB; j++) {
            const int64_t q = p0 + kB * 32 + j * 32 + lane;
            nxt[j] = q < P ? row[q] : T(0);
        }
#pragma unroll
        for (int j = 0; j < kB; j++) {
            const int64_t b = p0 + j * 32;
            if (b >= P) break;  // warp-uniform
            const T av = fabs(cur[j]);
            if (b + lane < P && av >= aes0) np++;
            // sequential sum in index order, as the reference's host loop;
            // unrolled, the shuffles run ahead of the chain of additions
            // (50 sets x 1,024 columns 16.5 -> 8.5 us)
            if (P - b >= 32) {
#pragma unroll
                for (int i = 0; i < 32; i++) sum = Exact<T>::add(sum, __shfl_sync(kFullMask, av, i));
            } else {
                const int n = (int)(P - b);
                for (int i = 0; i < n; i++) sum = Exact<T>::add(sum, __shfl_sync(kFullMask, av, i));
            }
        }
#pragma unroll
        for (int j = 0; j < kB; j++) cur[j] = nxt[j];
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) np += __shfl_xor_sync(kFullMask, np, o);
    if (lane == 0) {
        const T f = Exact<T>::div((T)P, sum);
        fac[warp] = f;
        out[warp] = es0;
        out[K + warp] = Exact<T>::mul(es0, f);
        out[2 * K + warp] = Exact<T>::div((T)np, (T)P);
    }
}

// extrema of the normalised scores per permutation column.  Each thread folds
// a chunk of sets for one column and merges it with an atomic max / min on
// the order-preserving radix image of the value (NaN skipped, as the
// reference's `<` / `>` updates skip it).  Radix image 0 ("empty" for the
// max) and all-ones ("empty" for the min) belong only to NaN bit patterns.
constexpr int kExtremaSets = 16;
template <class T>
__device__ __forceinline__ void stats_extrema_kernel_body(int bx, int by, const T* __restrict__ es, int K, int64_t ld, int64_t P, const T* __restrict__ fac,
                                     typename RadixKey<T>::U* __restrict__ mx,
                                     typename RadixKey<T>::U* __restrict__ mn) {
    using U = typename RadixKey<T>::U;
    const int64_t p = (int64_t)bx * blockDim.x + threadIdx.x;
    if (p >= P) return;
    const int k0 = by * kExtremaSets, k1 = min(K, k0 + kExtremaSets);
    T hi = -INFINITY, lo = INFINITY;
    for (int k = k0; k < k1; k++) {
        const T v = Exact<T>::mul(es[(int64_t)k * ld + p], fac[k]);
        hi = hi < v ? v : hi;
        lo = lo > v ? v : lo;
    }
    atomicMax(&mx[p], (U)RadixKey<T>::from(hi, false));
    atomicMin(&mn[p], (U)RadixKey<T>::from(lo, false));
}

template <class T>
__device__ __forceinline__ T radix_value(typename RadixKey<T>::U u);
template <>
__device__ __forceinline__ float radix_value<float>(uint32_t u) {
    u = (u & 0x80000000u) ? (u & 0x7fffffffu) : ~u;
    return __uint_as_float(u);
}
template <>
__device__ __forceinline__ double radix_value<double>(unsigned long long u) {
    u = (u & 0x8000000000000000ull) ? (u & 0x7fffffffffffffffull) : ~u;
    return __longlong_as_double((long long)u);
}

// one warp per set: FWER
template <class T>
__device__ __forceinline__ void stats_fwer_kernel_body(int bx, int K, int64_t P, const typename RadixKey<T>::U* __restrict__ mx,
                                  const typename RadixKey<T>::U* __restrict__ mn, T* __restrict__ out) {
    const int warp = (bx * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= K) return;
    const T score = out[K + warp];
    unsigned long long c = 0;
    if (score > T(0)) {
        for (int64_t p = lane; p < P; p += 32) c += radix_value<T>(mx[p]) >= score;
    } else {
        for (int64_t p = lane; p < P; p += 32) c += radix_value<T>(mn[p]) <= score;
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) c += __shfl_xor_sync(kFullMask, c, o);
    if (lane == 0) out[3 * K + warp] = Exact<T>::div((T)c, (T)P);
}

// ---------------------------------------------------------------------------
// FDR counts, exact, O(K*P) but for a short search in a slot of the observed
// keys (ObservedKeys).  Each side is handled as "key >= key*":
// positive side keys are the scores themselves (observed NES >= 0, null
// scores >= 0), negative side keys their negations (scores <= 0); a zero is on
// both sides, NaN on neither.
//   1. stats_fdr_obs_kernel: for every set, L = #{same-side observed keys <
//      its key} and the observed count #{>= key}; the observed keys are
//      scattered into ascending order at L + (#equal keys of lower index).
//   2. stats_fdr_hist_kernel: every null score is looked up among the sorted
//      observed keys of its side: t = #{observed keys <= it}, counted in H[t].
//   3. stats_fdr_suffix_kernel: S[i] = sum_{t >= i} H[t].
//   4. stats_fdr_final_kernel: #{null keys >= key*} = S[L + 1] (a null key v
//      satisfies v >= key* exactly when t(v) >= L + 1).
// Layout of the FDR part of the scratch (unsigned long long):
//   cnt_obs[K] | L[K] | sorted_pos[K] (T) | sorted_neg[K] (T) |
//   H_pos[K+2] | H_neg[K+2] (double weights) | totals[8]: [2], [3] observed
//   counts per side (u64), [4], [5] null weight per side (double)

template <class T>
__device__ __forceinline__ int side_of(T s) { return s > T(0) ? 0 : (s <= T(0) ? 1 : -1); }

// one warp per set; the lanes stride over the other sets and the counts are
// warp-reduced
template <class T>
__device__ __forceinline__ void stats_fdr_obs_kernel_body(int bx, int K, const T* __restrict__ out, unsigned long long* __restrict__ cnt_obs,
                                     unsigned long long* __restrict__ lcount, T* __restrict__ sorted_pos,
                                     T* __restrict__ sorted_neg, unsigned long long* __restrict__ totals) {
    const int k = (bx * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (k >= K) return;
    const T s = out[K + k];
    // membership in the two sorted arrays: o >= 0 (positive), o <= 0 (negative)
    for (int side = 0; side < 2; side++) {
        const bool in = side == 0 ? (s >= T(0)) : (s <= T(0));
        if (!in) continue;  // warp-uniform
        const T key = side == 0 ? s : -s;
        unsigned long long less = 0, eq_before = 0;
        for (int j = lane; j < K; j += 32) {
            const T o = out[K + j];
            const bool jin = side == 0 ? (o >= T(0)) : (o <= T(0));
            if (!jin) continue;
            const T oj = side == 0 ? o : -o;
            less += oj < key;
            eq_before += (oj == key) && (j < k);
        }
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) {
            less += __shfl_xor_sync(kFullMask, less, o);
            eq_before += __shfl_xor_sync(kFullMask, eq_before, o);
        }
        if (lane == 0) {
            (side == 0 ? sorted_pos : sorted_neg)[less + eq_before] = key;
            atomicAdd(&totals[2 + side], 1ull);
            // observed count on the set's own side: #{keys >= key} = m - less
            if (side_of(s) == side) lcount[k] = less;
        }
    }
    const int sd = side_of(s);
    if (sd >= 0) {
        const T key = sd == 0 ? s : -s;
        unsigned long long ge = 0;
        for (int j = lane; j < K; j += 32) {
            const T o = out[K + j];
            const bool jin = sd == 0 ? (o >= T(0)) : (o <= T(0));
            ge += jin && ((sd == 0 ? o : -o) >= key);
        }
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) ge += __shfl_xor_sync(kFullMask, ge, o);
        if (lane == 0) cnt_obs[k] = ge;
    }
}

template <class T>
__device__ __forceinline__ unsigned upper_bound_t(const T* a, unsigned lo, unsigned hi, T v) {
    while (lo < hi) {
        const unsigned mid = (lo + hi) >> 1;
        if (a[mid] <= v) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// The observed keys of both sides in shared memory, and for each side a table
// of kSlots slots of equal width from 0 to its largest key: the slot of a value
// never falls as the value grows, so that the keys of lower slots are below it
// and those of higher slots above, and the search is left with the keys of its
// own slot: 2 or 3 steps instead of 12 for 2,500 keys a side (the statistics of
// 2,000 sets x 1,000 columns 64 -> 59 us, of 1,000 x 1,000 47 -> 45; the weighted
// histograms of the adaptive test's six rounds 3,848 -> 3,566 us).
constexpr unsigned kSlots = 1024;
template <class T>
struct ObservedKeys {
    const T *pos, *neg;          // ascending
    unsigned npos, nneg;
    const unsigned short *tpos, *tneg;  // [kSlots + 1] keys in lower slots
    float spos, sneg;

    static __host__ __device__ size_t bytes(int K) {
        return (sizeof(T) * 2 * (size_t)K + 2 * (kSlots + 1) * sizeof(unsigned short) + 15) & ~(size_t)15;
    }
    static __device__ __forceinline__ unsigned slot(T v, float scale) {
        const float f = (float)v * scale;  // v >= 0; inf and NaN (0 * inf) go to the last and the first slot
        return f >= (float)kSlots ? kSlots - 1 : f > 0.f ? min((unsigned)f, kSlots - 1) : 0u;
    }
    // all threads of the block; `at`: bytes(K)
    __device__ __forceinline__ ObservedKeys(unsigned char* at, int K, const T* sorted_pos, const T* sorted_neg,
                                            unsigned n0, unsigned n1) {
        T* const k = reinterpret_cast<T*>(at);
        unsigned short* const t = reinterpret_cast<unsigned short*>(k + 2 * (size_t)K);
        pos = k;
        neg = k + n0;
        npos = n0;
        nneg = n1;
        tpos = t;
        tneg = t + kSlots + 1;
        for (unsigned i = threadIdx.x; i < n0; i += blockDim.x) k[i] = sorted_pos[i];
        for (unsigned i = threadIdx.x; i < n1; i += blockDim.x) k[n0 + i] = sorted_neg[i];
        __syncthreads();
        spos = fill(t, pos, n0);
        sneg = fill(t + kSlots + 1, neg, n1);
        __syncthreads();
    }
    static __device__ __forceinline__ float fill(unsigned short* t, const T* a, unsigned n) {
        const float scale = n ? (float)kSlots / (float)a[n - 1] : 0.f;
        for (unsigned q = threadIdx.x; q <= kSlots; q += blockDim.x) {  // keys whose slot is lower
            unsigned lo = 0, hi = n;
            while (lo < hi) {
                const unsigned mid = (lo + hi) >> 1;
                if (slot(a[mid], scale) < q) lo = mid + 1; else hi = mid;
            }
            t[q] = (unsigned short)lo;
        }
        return scale;
    }
    // observed keys <= v on a side
    __device__ __forceinline__ unsigned upto(bool up, T v) const {
        const unsigned q = slot(v, up ? spos : sneg);
        const unsigned short* const t = up ? tpos : tneg;
        return upper_bound_t(up ? pos : neg, t[q], t[q + 1], v);
    }
};

constexpr int kHistThreads = 1024;
constexpr int kHistCols = kHistThreads * 8;  // null columns per step
constexpr int kKeysMax = 65535;              // the table counts keys in 16 bits
// grid (sets, column chunks): block (b, c) bins the null scores of the sets
// b, b + gridDim.x, ... in the chunks c, c + gridDim.y, ... of kHistCols
// columns of each set's columns 1..m_k-1, m_k = min(n_k, hist_cols) (the
// adaptive test's intermediate rounds bin only the pilot columns: the same
// pooled null, each set's nulls weighted to equal total weight).  staged: 1 the
// sorted observed keys are in shared memory, 2 and counters of the bins: the
// block takes the sets of one length, which have one weight,
// and adds count times weight to the bins, in place of an FP64 atomic a score
// (the six rounds of an adaptive test of 5,000 sets x up to 20,000 columns 3,566
// -> 760 us).
template <class T>
__global__ void __launch_bounds__(kHistThreads)
stats_fdr_hist_kernel(const T* __restrict__ es, int K, int64_t ld, const int64_t* __restrict__ counts,
                      int64_t hist_cols, const T* __restrict__ fac, const T* sorted_pos, const T* sorted_neg,
                      double* __restrict__ hpos, double* __restrict__ hneg, unsigned long long* __restrict__ totals,
                      int staged) {
    extern __shared__ __align__(16) unsigned char hist_smem[];  // ObservedKeys, counters
    const unsigned npos = (unsigned)totals[2], nneg = (unsigned)totals[3];
    double* wtot = reinterpret_cast<double*>(totals + 4);
    double cpos = 0.0, cneg = 0.0;
    // the scores of set k's first n columns, bin(up, value) for each: column
    // c0 + t, c0 + t + step, ... of a chunk that starts at c0
    auto row_scores = [&](int64_t k, int64_t n, int t, int step, auto&& bin) {
        const T f = fac[k];
        const T* row = es + k * ld;
        for (int64_t c0 = 1 + (int64_t)blockIdx.y * kHistCols; c0 < n; c0 += (int64_t)gridDim.y * kHistCols) {
            const int64_t c1 = c0 + kHistCols < n ? c0 + kHistCols : n;
            for (int64_t p = c0 + t; p < c1; p += step) {
                const T v = Exact<T>::mul(row[p], f);
                if (v >= T(0)) bin(true, v);
                if (v <= T(0)) bin(false, -v);
            }
        }
    };
    auto columns = [&](int64_t k) {
        const int64_t n = counts ? counts[k] : ld;
        return n < hist_cols ? n : hist_cols;
    };
    auto weight = [&](int64_t n) { return counts ? (double)(ld - 1) / (double)(n - 1) : 1.0; };
    // a score at a time; sets of few columns by warps
    // (40,000 sets x 10 columns 2,699 -> 2,328 us; 10,000 in double x 400 2,471 -> 2,494)
    auto one_by_one = [&](auto&& upto) {
        const bool warps = hist_cols <= 256;
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const int t = warps ? lane : (int)threadIdx.x, step = warps ? 32 : kHistThreads;
        const int64_t stride = (int64_t)gridDim.x * (warps ? kHistThreads / 32 : 1);
        for (int64_t k = blockIdx.x + (warps ? (int64_t)warp * gridDim.x : 0); k < K; k += stride) {
            const int64_t n = columns(k);
            if (n < 2) continue;
            const double w = weight(n);
            row_scores(k, n, t, step, [&](bool pos, T v) {
                (pos ? cpos : cneg) += w;
                atomicAdd((pos ? hpos : hneg) + upto(pos, v), w);
            });
        }
    };
    if (staged == 2) {
        const ObservedKeys<T> keys(hist_smem, K, sorted_pos, sorted_neg, npos, nneg);
        unsigned* const h = reinterpret_cast<unsigned*>(hist_smem + ObservedKeys<T>::bytes(K));  // 2 (K + 2)
        const int W = 2 * (K + 2);
        for (int i = threadIdx.x; i < W; i += kHistThreads) h[i] = 0u;
        int64_t n = 0;  // the columns of the group before
        while (true) {
            int64_t next = INT64_MAX;
            for (int64_t k = blockIdx.x; k < K; k += gridDim.x) {
                const int64_t m = columns(k);
                if (m > n && m < next) next = m;
            }
            if (next == INT64_MAX) break;  // the same in every thread
            n = next;
            if (n < 2) continue;
            __syncthreads();  // the counters are clear
            unsigned up = 0u, down = 0u;
            for (int64_t k = blockIdx.x; k < K; k += gridDim.x) {
                if (columns(k) != n) continue;
                row_scores(k, n, (int)threadIdx.x, kHistThreads, [&](bool pos, T v) {
                    (pos ? up : down)++;
                    atomicAdd(&h[(pos ? 0 : K + 2) + keys.upto(pos, v)], 1u);
                });
            }
            __syncthreads();
            const double w = weight(n);
            cpos += (double)up * w;
            cneg += (double)down * w;
            for (int i = threadIdx.x; i < W; i += kHistThreads) {
                const unsigned c = h[i];
                if (c) {
                    h[i] = 0u;
                    atomicAdd(i < K + 2 ? &hpos[i] : &hneg[i - (K + 2)], (double)c * w);
                }
            }
        }
    } else if (staged == 1) {
        const ObservedKeys<T> keys(hist_smem, K, sorted_pos, sorted_neg, npos, nneg);
        one_by_one([&](bool pos, T v) { return keys.upto(pos, v); });
    } else {
        one_by_one([&](bool pos, T v) {
            return upper_bound_t(pos ? sorted_pos : sorted_neg, 0u, pos ? npos : nneg, v);
        });
    }
    for (int o = 16; o >= 1; o >>= 1) {
        cpos += __shfl_xor_sync(kFullMask, cpos, o);
        cneg += __shfl_xor_sync(kFullMask, cneg, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (cpos != 0.0) atomicAdd(&wtot[0], cpos);
        if (cneg != 0.0) atomicAdd(&wtot[1], cneg);
    }
}

// Dense form (every set has all ld columns, unit weights): block b bins an
// equal contiguous share of the K x (ld - 1) null scores (row-major, column
// 0 excluded) into shared-memory integer histograms of both sides, against
// the sorted observed keys staged beside them, and adds its bins that are not
// empty to the global ones: exact integer counts, the same in any order.
constexpr int kDenseHistThreads = 1024;
constexpr size_t kDenseHistSmemMax = 96 * 1024;
constexpr int kDenseHistShare = 1024;  // scores of a block, at least: one a thread
template <class T>
__device__ __forceinline__ void
stats_fdr_hist_dense_body(int bx, int gx, const T* __restrict__ es, int K, int64_t ld, const T* __restrict__ fac,
                          const T* __restrict__ sorted_pos, const T* __restrict__ sorted_neg,
                          const unsigned long long* __restrict__ totals, unsigned long long* __restrict__ bins) {
    extern __shared__ __align__(16) unsigned char dense_smem[];
    const int W = 2 * (K + 2);
    unsigned* h = reinterpret_cast<unsigned*>(dense_smem);  // W counters
    for (int i = threadIdx.x; i < W; i += kDenseHistThreads) h[i] = 0u;
    const ObservedKeys<T> keys(dense_smem + (((size_t)W * 4 + 15) & ~(size_t)15), K, sorted_pos, sorted_neg,
                               (unsigned)totals[2], (unsigned)totals[3]);
    const int64_t cols = ld - 1;
    const int64_t total = (int64_t)K * cols;
    const int64_t lo = total * bx / gx, hi = total * (bx + 1) / gx;
    // a score a thread whatever row it is in: with few columns a row at a time
    // leaves most threads idle (1,000 sets x 2 columns 395 -> 31 us, 10 columns
    // 110 -> 31, 100 39 -> 31, 400 41 -> 39)
    if (cols <= kDenseHistThreads / 2) {  // then fewer than 2^32 scores
        for (uint32_t i = (uint32_t)lo + threadIdx.x; i < (uint32_t)hi; i += kDenseHistThreads) {
            const uint32_t k = i / (uint32_t)cols, c = i - k * (uint32_t)cols;
            const T v = Exact<T>::mul(es[k * ld + 1 + c], fac[k]);
            if (v >= T(0)) atomicAdd(&h[keys.upto(true, v)], 1u);
            if (v <= T(0)) atomicAdd(&h[(K + 2) + keys.upto(false, -v)], 1u);
        }
    } else {
        int64_t k = lo / cols;
        int64_t c = lo - k * cols;  // column - 1 within row k
        for (int64_t i = lo; i < hi;) {
            const int64_t run = (cols - c) < (hi - i) ? (cols - c) : (hi - i);  // rest of row k in the share
            const T f = fac[k];
            const T* row = es + k * ld + 1 + c;
            for (int64_t j = threadIdx.x; j < run; j += kDenseHistThreads) {
                const T v = Exact<T>::mul(row[j], f);
                if (v >= T(0)) atomicAdd(&h[keys.upto(true, v)], 1u);
                if (v <= T(0)) atomicAdd(&h[(K + 2) + keys.upto(false, -v)], 1u);
            }
            i += run;
            k++;
            c = 0;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < W; i += kDenseHistThreads)
        if (h[i]) atomicAdd(&bins[i], (unsigned long long)h[i]);
}

template <class T>
size_t dense_hist_smem(int K) {
    const size_t W = 2 * ((size_t)K + 2) + 2;
    return ((W * 4 + 15) & ~(size_t)15) + ObservedKeys<T>::bytes(K);
}
// the counters and the keys fit half of an SM's shared memory
template <class T>
bool dense_applies(int K) {
    return (((2 * ((size_t)K + 2) + 2) * 4 + 15) & ~(size_t)15) + 2 * sizeof(T) * (size_t)K <= kDenseHistSmemMax;
}
// blocks of the dense histogram (0: the dense form does not apply): two to
// an SM, fewer where a share would not pay for staging the observed keys
template <class T>
int dense_hist_blocks(int K, int64_t ld, int sms) {
    if (!dense_applies<T>(K)) return 0;
    const int64_t shares = ((int64_t)K * (ld - 1) + kDenseHistShare - 1) / kDenseHistShare;
    const int64_t want = 2 * (int64_t)(sms > 0 ? sms : 1);
    return (int)(shares < 1 ? 1 : shares < want ? shares : want);
}

// in-place suffix sums of the two histograms (one block each)
__device__ __forceinline__ void stats_fdr_suffix_kernel_body(int bx, double* __restrict__ hpos, double* __restrict__ hneg,
                                        const unsigned long long* __restrict__ totals) {
    double* h = bx == 0 ? hpos : hneg;
    const unsigned n = (unsigned)totals[2 + bx] + 1;  // bins 0..m
    __shared__ double carry;
    __shared__ double wsum[32];
    if (threadIdx.x == 0) carry = 0.0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    // walk from the top bin down in chunks of blockDim.x
    for (int64_t top = (int64_t)n - 1; top >= 0; top -= blockDim.x) {
        const int64_t i = top - threadIdx.x;
        double v = i >= 0 ? h[i] : 0.0;
        for (int o = 1; o < 32; o <<= 1) {
            const double y = __shfl_up_sync(kFullMask, v, o);
            if (lane >= o) v += y;
        }
        if (lane == 31) wsum[warp] = v;
        __syncthreads();
        double before = carry;
        for (int w = 0; w < warp; w++) before += wsum[w];
        if (i >= 0) h[i] = v + before;
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (int w = 0; w < nw; w++) t += wsum[w];
            carry += t;
        }
        __syncthreads();
    }
}

template <class T>
__device__ __forceinline__ void stats_fdr_final_kernel_body(int bx, int K, const unsigned long long* __restrict__ cnt_obs,
                                       const unsigned long long* __restrict__ lcount,
                                       const double* __restrict__ spos, const double* __restrict__ sneg,
                                       const unsigned long long* __restrict__ totals, T* __restrict__ out) {
    const int k = bx * blockDim.x + threadIdx.x;
    if (k >= K) return;
    const T s = out[K + k];
    T q;
    if (!(s == s)) {
        q = s;
    } else {
        const bool up = s > T(0);
        const unsigned long long L = lcount[k];
        const unsigned long long m = up ? totals[2] : totals[3];
        const double* wtot = reinterpret_cast<const double*>(totals + 4);
        const double c_null = L + 1 <= m ? (up ? spos : sneg)[L + 1] : 0.0;
        const double null_side = up ? wtot[0] : wtot[1];
        const double obs_side = (double)m;
        const double fn = null_side > 0 ? c_null / null_side : 0.0;
        const double fo = (double)cnt_obs[k] / obs_side;
        const double r = fn / fo;
        q = (T)(r < 1.0 ? r : 1.0);
    }
    out[4 * K + k] = q;
}

// the statistics scratch of K sets with FWER over p_fwer columns
template <class T>
struct RaggedLayout {
    using U = typename RadixKey<T>::U;
    T* fac;
    U* mx;
    U* mn;
    unsigned long long* cnt_obs;
    unsigned long long* lcount;
    T* sorted_pos;
    T* sorted_neg;
    double* hpos;
    double* hneg;
    unsigned long long* totals;
    unsigned long long* bins;  // dense form: null scores per bin, 2(K+2)
    __host__ __device__ RaggedLayout(void* scratch, int K, int64_t p_fwer) {
        unsigned char* s = static_cast<unsigned char*>(scratch);
        auto align16 = [](size_t x) { return (x + 15) & ~(size_t)15; };
        fac = reinterpret_cast<T*>(s);
        mx = reinterpret_cast<U*>(fac + K);
        mn = mx + p_fwer;
        size_t off = align16(sizeof(T) * ((size_t)K + 2 * (size_t)p_fwer));
        cnt_obs = reinterpret_cast<unsigned long long*>(s + off);
        lcount = cnt_obs + K;
        off = align16(off + sizeof(unsigned long long) * 2 * (size_t)K);
        sorted_pos = reinterpret_cast<T*>(s + off);
        sorted_neg = sorted_pos + K;
        off = align16(off + sizeof(T) * 2 * (size_t)K);
        hpos = reinterpret_cast<double*>(s + off);
        hneg = hpos + (K + 2);
        totals = reinterpret_cast<unsigned long long*>(hneg + (K + 2));
        bins = reinterpret_cast<unsigned long long*>(s + align16(off + sizeof(double) * (2 * ((size_t)K + 2) + 8)));
    }
};

// ---- the kernels of one statistics run (solo) --------------------------------
template <class T>
__global__ void stats_set_kernel(const T* __restrict__ es, int K, int64_t ld, const int64_t* __restrict__ counts,
                                 T* __restrict__ out, T* __restrict__ fac) {
    stats_set_kernel_body<T>(blockIdx.x, es, K, ld, counts, out, fac);
}
template <class T>
__global__ void stats_extrema_kernel(const T* __restrict__ es, int K, int64_t ld, int64_t P, const T* __restrict__ fac,
                                     typename RadixKey<T>::U* __restrict__ mx, typename RadixKey<T>::U* __restrict__ mn) {
    stats_extrema_kernel_body<T>(blockIdx.x, blockIdx.y, es, K, ld, P, fac, mx, mn);
}
template <class T>
__global__ void stats_fwer_kernel(int K, int64_t P, const typename RadixKey<T>::U* __restrict__ mx,
                                  const typename RadixKey<T>::U* __restrict__ mn, T* __restrict__ out) {
    stats_fwer_kernel_body<T>(blockIdx.x, K, P, mx, mn, out);
}
template <class T>
__global__ void stats_fdr_obs_kernel(int K, const T* __restrict__ out, unsigned long long* __restrict__ cnt_obs,
                                     unsigned long long* __restrict__ lcount, T* __restrict__ sorted_pos,
                                     T* __restrict__ sorted_neg, unsigned long long* __restrict__ totals) {
    stats_fdr_obs_kernel_body<T>(blockIdx.x, K, out, cnt_obs, lcount, sorted_pos, sorted_neg, totals);
}
__global__ void stats_fdr_suffix_kernel(double* __restrict__ hpos, double* __restrict__ hneg,
                                        const unsigned long long* __restrict__ totals) {
    stats_fdr_suffix_kernel_body(blockIdx.x, hpos, hneg, totals);
}
template <class T>
__global__ void stats_fdr_final_kernel(int K, const unsigned long long* __restrict__ cnt_obs,
                                       const unsigned long long* __restrict__ lcount,
                                       const double* __restrict__ spos, const double* __restrict__ sneg,
                                       const unsigned long long* __restrict__ totals, T* __restrict__ out) {
    stats_fdr_final_kernel_body<T>(blockIdx.x, K, cnt_obs, lcount, spos, sneg, totals, out);
}

// ---- the dense form in four steps --------------------------------------------
// Every set has all its columns.  Independent kernels of the list above share
// a launch (blocks of different kinds), the buffers are cleared by the first:
//   1. factors, NES, NP; histogram, totals and extrema cleared
//   2. extrema per column; counts and order of the observed scores
//   3. null histogram; FWER
//   4. suffix sums and q
// (Eight launches and three memsets before: 70 us at 50 sets x 1,024
// permutations, most of it launches, one thread adding up 300 partial rows
// and FP64 prefix sums; the counts are integers here.)
struct DenseDims {
    int K, rows;        // sets; blocks of the histogram
    int64_t ld, p_fwer;
    __host__ __device__ int set_blocks() const { return (K + 7) / 8; }
    __host__ __device__ int64_t init() const { return p_fwer > 2 * (K + 2) + 8 ? p_fwer : 2 * (K + 2) + 8; }
    __host__ __device__ int extrema_x() const { return (int)((p_fwer + 127) / 128); }
    __host__ __device__ int64_t extrema_blocks() const {
        return (int64_t)extrema_x() * ((K + kExtremaSets - 1) / kExtremaSets);
    }
    __host__ __device__ int64_t step2_blocks() const { return extrema_blocks() + (K + 3) / 4; }
    __host__ __device__ int step3_blocks() const { return rows + (K + kDenseHistThreads / 32 - 1) / (kDenseHistThreads / 32); }
};

template <class T>
__device__ __forceinline__ void dense_step1(int64_t bx, int64_t gx, const DenseDims& d, const T* es, T* out,
                                            const RaggedLayout<T>& L) {
    using U = typename RadixKey<T>::U;
    for (int64_t i = bx * blockDim.x + threadIdx.x; i < d.init(); i += gx * blockDim.x) {
        if (i < 2 * (d.K + 2)) L.bins[i] = 0ull;
        else if (i < 2 * (d.K + 2) + 8) L.totals[i - 2 * (d.K + 2)] = 0ull;
        if (i < d.p_fwer) {
            L.mx[i] = U(0);
            L.mn[i] = ~U(0);
        }
    }
    if (bx < d.set_blocks()) stats_set_kernel_body<T>((int)bx, es, d.K, d.ld, nullptr, out, L.fac);
}
template <class T>
__device__ __forceinline__ void dense_step2(int64_t bx, const DenseDims& d, const T* es, const T* out,
                                            const RaggedLayout<T>& L) {
    const int64_t ext = d.extrema_blocks();
    if (bx < ext) {
        const int gx = d.extrema_x();
        stats_extrema_kernel_body<T>((int)(bx % gx), (int)(bx / gx), es, d.K, d.ld, d.p_fwer, L.fac, L.mx, L.mn);
    } else {
        stats_fdr_obs_kernel_body<T>((int)(bx - ext), d.K, out, L.cnt_obs, L.lcount, L.sorted_pos, L.sorted_neg,
                                     L.totals);
    }
}
template <class T>
__device__ __forceinline__ void dense_step3(int bx, const DenseDims& d, const T* es, T* out,
                                            const RaggedLayout<T>& L) {
    if (bx < d.rows)
        stats_fdr_hist_dense_body<T>(bx, d.rows, es, d.K, d.ld, L.fac, L.sorted_pos, L.sorted_neg, L.totals, L.bins);
    else
        stats_fwer_kernel_body<T>(bx - d.rows, d.K, d.p_fwer, L.mx, L.mn, out);
}
// q of kQSets sets on one side (0: positive, 1: negative).  Every block sums
// the side's bins for itself, in shared memory: the quotients are what takes
// time (four FP64 divisions a set; one block for 1,000 sets: 18 us), and a
// warp to each quarter of the SM is as many as they keep busy.
constexpr int kQSets = 128;
template <class T>
__device__ __forceinline__ void dense_step4(int bx, int side, const DenseDims& d, T* out, const RaggedLayout<T>& L) {
    extern __shared__ __align__(16) unsigned long long above_bin[];  // [K + 2] scores in bin i or above
    __shared__ unsigned long long carry, wsum[32];
    const unsigned long long* const h = L.bins + side * (d.K + 2);
    const int m = (int)L.totals[2 + side], n = m + 1;  // bins 0..m
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 0ull;
    __syncthreads();
    for (int top = n - 1; top >= 0; top -= (int)blockDim.x) {  // from the top bin down
        const int i = top - (int)threadIdx.x;
        unsigned long long v = i >= 0 ? h[i] : 0ull;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(kFullMask, v, o);
            if (lane >= o) v += y;
        }
        if (lane == 31) wsum[warp] = v;
        __syncthreads();
        unsigned long long w = wsum[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(kFullMask, w, o);
            if (lane >= o) w += y;
        }
        const unsigned long long before = warp > 0 ? __shfl_sync(kFullMask, w, (warp + 31) & 31) : 0ull;
        const unsigned long long all = __shfl_sync(kFullMask, w, 31), c = carry;
        if (i >= 0) above_bin[i] = v + before + c;
        __syncthreads();
        if (threadIdx.x == 0) carry = c + all;
        __syncthreads();
    }
    const double null_side = (double)carry;
    const int k = bx * kQSets + (int)threadIdx.x;
    if (threadIdx.x >= kQSets || k >= d.K) return;
    const T s = out[d.K + k];
    const bool up = s > T(0);
    if (!(s == s)) {
        if (side == 0) out[4 * d.K + k] = s;
    } else if (up == (side == 0)) {
        const unsigned long long above = L.lcount[k] + 1;
        const double c_null = above <= (unsigned long long)m ? (double)above_bin[above] : 0.0;
        const double fn = null_side > 0 ? c_null / null_side : 0.0;
        const double fo = (double)L.cnt_obs[k] / (double)m;
        const double r = fn / fo;
        out[4 * d.K + k] = (T)(r < 1.0 ? r : 1.0);
    }
}
inline size_t dense_q_smem(int K) { return sizeof(unsigned long long) * ((size_t)K + 2); }

template <class T>
__global__ void __launch_bounds__(256) stats_dense1_kernel(DenseDims d, const T* es, T* out, RaggedLayout<T> L) {
    dense_step1<T>(blockIdx.x, gridDim.x, d, es, out, L);
}
template <class T>
__global__ void __launch_bounds__(128) stats_dense2_kernel(DenseDims d, const T* es, T* out, RaggedLayout<T> L) {
    dense_step2<T>(blockIdx.x, d, es, out, L);
}
template <class T>
__global__ void __launch_bounds__(kDenseHistThreads)
stats_dense3_kernel(DenseDims d, const T* es, T* out, RaggedLayout<T> L) {
    dense_step3<T>(blockIdx.x, d, es, out, L);
}
template <class T>
__global__ void __launch_bounds__(1024) stats_dense4_kernel(DenseDims d, T* out, RaggedLayout<T> L) {
    dense_step4<T>(blockIdx.x, blockIdx.y, d, out, L);
}

// many instances at once: blockIdx.z = the instance; grids are sized for the
// largest and the blocks beyond an instance's own extent return at once
template <class T>
__device__ __forceinline__ DenseDims dims_of(const StatsTask<T>& t) { return DenseDims{t.K, t.rows, t.P, t.P}; }
template <class T>
__global__ void __launch_bounds__(256) stats_dense1_multi(const StatsTask<T>* __restrict__ tasks) {
    const StatsTask<T> t = tasks[blockIdx.z];
    const RaggedLayout<T> L(t.scratch, t.K, t.P);
    dense_step1<T>(blockIdx.x, gridDim.x, dims_of(t), t.es, t.stats, L);
}
template <class T>
__global__ void __launch_bounds__(128) stats_dense2_multi(const StatsTask<T>* __restrict__ tasks) {
    const StatsTask<T> t = tasks[blockIdx.z];
    const DenseDims d = dims_of(t);
    if ((int64_t)blockIdx.x >= d.step2_blocks()) return;
    const RaggedLayout<T> L(t.scratch, t.K, t.P);
    dense_step2<T>(blockIdx.x, d, t.es, t.stats, L);
}
template <class T>
__global__ void __launch_bounds__(kDenseHistThreads) stats_dense3_multi(const StatsTask<T>* __restrict__ tasks) {
    const StatsTask<T> t = tasks[blockIdx.z];
    const DenseDims d = dims_of(t);
    if ((int)blockIdx.x >= d.step3_blocks()) return;  // the whole block: before any barrier
    const RaggedLayout<T> L(t.scratch, t.K, t.P);
    dense_step3<T>(blockIdx.x, d, t.es, t.stats, L);
}
template <class T>
__global__ void __launch_bounds__(1024) stats_dense4_multi(const StatsTask<T>* __restrict__ tasks) {
    const StatsTask<T> t = tasks[blockIdx.z];
    if ((int)blockIdx.x * kQSets >= t.K) return;  // the whole block: before any barrier
    const RaggedLayout<T> L(t.scratch, t.K, t.P);
    dense_step4<T>(blockIdx.x, blockIdx.y, dims_of(t), t.stats, L);
}

// Lower bound of every set's FDR q after the statistics (adaptive stopping):
// the set's |NES| may lie anywhere in [|NES|, key], key = |NES| (1 + z cv /
// sqrt(n)) -- z standard errors of its normalising mean, cv the coefficient
// of variation of its n scores |S| (sums[k] = sum |S|, sums[K + k] = sum
// S^2).  q(x) = (null weight >= x / null weight of the side) / (#observed >=
// x / m) is not monotone in x, so the bound takes the least numerator and
// the largest denominator over the interval: with i_up observed keys below
// key, at least S[i_up + 1] null weight lies at or above key (the nulls at or
// above the next observed key); with i_lo observed keys below |NES|, at most
// m - i_lo observed keys lie at or above |NES|:
//   q >= (S[i_up + 1] / null weight of the side) / (max(m - i_lo, 1) / m).
// NaN or zero NES: 0 (no bound).
template <class T>
__global__ void stats_fdr_bound_kernel(int K, const T* __restrict__ stats, const int64_t* __restrict__ counts,
                                       const double* __restrict__ sums, double z, const T* __restrict__ sorted_pos,
                                       const T* __restrict__ sorted_neg, const double* __restrict__ spos,
                                       const double* __restrict__ sneg, const unsigned long long* __restrict__ totals,
                                       float* __restrict__ qlow, float* __restrict__ qhigh) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= K) return;
    const double s = (double)stats[K + k];
    float out = 0.f, out_hi = 1.f;
    const double n = (double)counts[k];
    if (s == s && s != 0.0 && n > 0) {
        const bool up = s > 0.0;
        const double m = sums[k] / n;
        const double var = fmax(sums[K + k] / n - m * m, 0.0);
        const double cv = m > 0.0 ? sqrt(var) / m : INFINITY;
        const double key = fabs(s) * (1.0 + z * cv / sqrt(n));
        const unsigned mcount = (unsigned)(up ? totals[2] : totals[3]);
        if (key < INFINITY && mcount > 0) {
            const T* keys = up ? sorted_pos : sorted_neg;
            auto below = [&](double x) {  // #{keys < x}
                unsigned lo = 0, hi = mcount;
                while (lo < hi) {
                    const unsigned mid = (lo + hi) >> 1;
                    if ((double)keys[mid] < x) lo = mid + 1; else hi = mid;
                }
                return lo;
            };
            const unsigned i_up = below(key), i_lo = below(fabs(s));
            const double c_null = i_up + 1 <= mcount ? (up ? spos : sneg)[i_up + 1] : 0.0;
            const double wtot = reinterpret_cast<const double*>(totals + 4)[up ? 0 : 1];
            const double fn = wtot > 0.0 ? c_null / wtot : 0.0;
            const double obs = (double)(mcount - i_lo > 0 ? mcount - i_lo : 1u);
            const double r = fn / (obs / (double)mcount);
            out = (float)(r < 1.0 ? r : 1.0);
            if (qhigh) {
                // upper bound: the most null weight (at the interval's bottom,
                // |NES| pulled inward) over the fewest observed keys (at or
                // above its top; the set's own key is one of them)
                const double key_in = fabs(s) * fmax(1.0 - z * cv / sqrt(n), 0.0);
                const unsigned j_in = below(key_in);
                const double c_in = j_in <= mcount ? (up ? spos : sneg)[j_in] : 0.0;
                const double fn_hi = wtot > 0.0 ? c_in / wtot : 1.0;
                const double obs_hi = (double)(mcount - i_up > 0 ? mcount - i_up : 1u);
                const double rh = fn_hi / (obs_hi / (double)mcount);
                out_hi = (float)(rh < 1.0 ? rh : 1.0);
            }
        }
    }
    qlow[k] = out;
    if (qhigh) qhigh[k] = out_hi;
}

}  // namespace

template <class T>
cudaError_t launch_fdr_bound(int K, int64_t p_fwer, const T* stats, const int64_t* counts, const double* sums,
                             double z, const void* scratch, float* qlow, cudaStream_t st, float* qhigh) {
    if (K <= 0) return cudaSuccess;
    const RaggedLayout<T> L(const_cast<void*>(scratch), K, p_fwer);
    stats_fdr_bound_kernel<T><<<(K + 255) / 256, 256, 0, st>>>(K, stats, counts, sums, z, L.sorted_pos, L.sorted_neg,
                                                               L.hpos, L.hneg, L.totals, qlow, qhigh);
    launches_add(1);
    return cudaGetLastError();
}
template cudaError_t launch_fdr_bound<float>(int, int64_t, const float*, const int64_t*, const double*, double,
                                             const void*, float*, cudaStream_t, float*);
template cudaError_t launch_fdr_bound<double>(int, int64_t, const double*, const int64_t*, const double*, double,
                                              const void*, float*, cudaStream_t, float*);

template <class T>
size_t stats_scratch_bytes(int K, int64_t P) {
    // + room for the dense histogram (2(K+2) 64-bit bins; what its rows of
    // partial counts once took, which callers of the C entry have allowed for)
    const size_t W = 2 * ((size_t)K + 2) + 2;
    const size_t dense = dense_applies<T>(K) ? ((size_t(1) << 20) / (4 * W)) * 4 * W + 16 : 0;
    return StatsScratch::bytes(K, P, sizeof(T)) + 256 + dense;
}
template size_t stats_scratch_bytes<float>(int, int64_t);
template size_t stats_scratch_bytes<double>(int, int64_t);

template <class T>
cudaError_t launch_stats_ragged(const T* es, int K, int64_t ld, const int64_t* counts, int64_t p_fwer, T* stats,
                                void* scratch, cudaStream_t st, int64_t hist_cols) {
    if (hist_cols <= 0 || hist_cols > ld) hist_cols = ld;
    if (K <= 0 || ld <= 0 || p_fwer <= 0 || p_fwer > ld) return K <= 0 ? cudaSuccess : cudaErrorInvalidValue;
    using U = typename RadixKey<T>::U;
    const RaggedLayout<T> L(scratch, K, p_fwer);
    int dev = 0, max_smem = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (!counts && ld > 1 && hist_cols == ld) {
        const DenseDims d{K, dense_hist_blocks<T>(K, ld, sms), ld, p_fwer};
        if (d.rows > 0 && d.step2_blocks() <= INT32_MAX) {
            const size_t smem = dense_hist_smem<T>(K);
            cudaError_t e = allow_smem(stats_dense3_kernel<T>, smem);
            if (e == cudaSuccess) e = allow_smem(stats_dense4_kernel<T>, dense_q_smem(K));
            if (e != cudaSuccess) return e;
            const int64_t clear = (d.init() + 255) / 256;  // blocks that clear, at most one to an SM more
            const int b1 = d.set_blocks() > sms ? d.set_blocks() : (int)(clear < sms ? std::max<int64_t>(clear, d.set_blocks()) : sms);
            stats_dense1_kernel<T><<<b1, 256, 0, st>>>(d, es, stats, L);
            stats_dense2_kernel<T><<<(unsigned)d.step2_blocks(), 128, 0, st>>>(d, es, stats, L);
            stats_dense3_kernel<T><<<d.step3_blocks(), kDenseHistThreads, smem, st>>>(d, es, stats, L);
            stats_dense4_kernel<T><<<dim3((K + kQSets - 1) / kQSets, 2), 1024, dense_q_smem(K), st>>>(d, stats, L);
            launches_add(4);
            return cudaGetLastError();
        }
    }
    T* fac = L.fac;
    U* mx = L.mx;
    U* mn = L.mn;
    unsigned long long* cnt_obs = L.cnt_obs;
    unsigned long long* lcount = L.lcount;
    T* sorted_pos = L.sorted_pos;
    T* sorted_neg = L.sorted_neg;
    double* hpos = L.hpos;
    double* hneg = L.hneg;
    unsigned long long* totals = L.totals;
    cudaError_t e = cudaMemsetAsync(hpos, 0, sizeof(double) * (2 * ((size_t)K + 2) + 8), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(mx, 0x00, sizeof(U) * (size_t)p_fwer, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(mn, 0xff, sizeof(U) * (size_t)p_fwer, st);
    if (e != cudaSuccess) return e;
    const int wpb = 8;  // warps per block
    stats_set_kernel<T><<<(K + wpb - 1) / wpb, wpb * 32, 0, st>>>(es, K, ld, counts, stats, fac);
    stats_extrema_kernel<T><<<dim3((unsigned)((p_fwer + 127) / 128), (K + kExtremaSets - 1) / kExtremaSets), 128, 0,
                              st>>>(es, K, ld, p_fwer, fac, mx, mn);
    stats_fwer_kernel<T><<<(K + wpb - 1) / wpb, wpb * 32, 0, st>>>(K, p_fwer, mx, mn, stats);
    stats_fdr_obs_kernel<T><<<(K + wpb - 1) / wpb, wpb * 32, 0, st>>>(K, stats, cnt_obs, lcount, sorted_pos,
                                                                       sorted_neg, totals);
    if (ld > 1) {
        // Two blocks to an SM where the keys leave room for it, each over many
        // sets, so that staging the keys pays; few sets are split by columns.
        const size_t room = max_smem > 1024 ? (size_t)max_smem - 1024 : 0, keys = ObservedKeys<T>::bytes(K);
        const size_t counters = 2 * ((size_t)K + 2) * sizeof(unsigned);
        const int staged = 2 * (int64_t)K > kKeysMax || keys > room ? 0 : keys + counters > room ? 1 : 2;
        const size_t smem = staged == 0 ? 0 : staged == 1 ? keys : keys + counters;
        const int64_t want = 2 * (int64_t)sms, chunks = (hist_cols - 1 + kHistCols - 1) / kHistCols;
        const int64_t x = K < want ? K : want, y = std::min<int64_t>(std::max<int64_t>(1, 2 * want / x), chunks);
        auto kern = stats_fdr_hist_kernel<T>;
        e = allow_smem(kern, smem);
        if (e != cudaSuccess) return e;
        kern<<<dim3((unsigned)x, (unsigned)(y > 0 ? y : 1)), kHistThreads, smem, st>>>(
            es, K, ld, counts, hist_cols, fac, sorted_pos, sorted_neg, hpos, hneg, totals, staged);
    }
    stats_fdr_suffix_kernel<<<2, 1024, 0, st>>>(hpos, hneg, totals);
    stats_fdr_final_kernel<T><<<(K + 255) / 256, 256, 0, st>>>(K, cnt_obs, lcount, hpos, hneg, totals, stats);
    launches_add(ld > 1 ? 7 : 6);
    return cudaGetLastError();
}
template cudaError_t launch_stats_ragged<float>(const float*, int, int64_t, const int64_t*, int64_t, float*, void*,
                                                cudaStream_t, int64_t);
template cudaError_t launch_stats_ragged<double>(const double*, int, int64_t, const int64_t*, int64_t, double*, void*,
                                                 cudaStream_t, int64_t);

template <class T>
int stats_multi_rows(int K, int64_t P) {
    if (K <= 0 || P < 2) return 0;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return dense_hist_blocks<T>(K, P, sms);
}
template int stats_multi_rows<float>(int, int64_t);
template int stats_multi_rows<double>(int, int64_t);

template <class T>
cudaError_t launch_stats_multi(const StatsTask<T>* d_tasks, const StatsTask<T>* h_tasks, int n, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    if (n > 65535) return cudaErrorInvalidValue;
    int b1 = 1, b3 = 1, Kmax = 1;
    int64_t b2 = 1;
    size_t smem = 0;
    for (int i = 0; i < n; i++) {
        const StatsTask<T>& t = h_tasks[i];
        if (t.rows <= 0 || t.P < 2) return cudaErrorInvalidValue;  // the dense form only
        const DenseDims d{t.K, t.rows, t.P, t.P};
        b1 = std::max(b1, d.set_blocks());
        b2 = std::max(b2, d.step2_blocks());
        b3 = std::max(b3, d.step3_blocks());
        smem = std::max(smem, dense_hist_smem<T>(t.K));
        Kmax = std::max(Kmax, t.K);
    }
    if (b2 > INT32_MAX) return cudaErrorInvalidValue;
    const unsigned z = (unsigned)n;
    cudaError_t e = allow_smem(stats_dense3_multi<T>, smem);
    if (e == cudaSuccess) e = allow_smem(stats_dense4_multi<T>, dense_q_smem(Kmax));
    if (e != cudaSuccess) return e;
    stats_dense1_multi<T><<<dim3((unsigned)b1, 1, z), 256, 0, st>>>(d_tasks);
    stats_dense2_multi<T><<<dim3((unsigned)b2, 1, z), 128, 0, st>>>(d_tasks);
    stats_dense3_multi<T><<<dim3((unsigned)b3, 1, z), kDenseHistThreads, smem, st>>>(d_tasks);
    stats_dense4_multi<T><<<dim3((Kmax + kQSets - 1) / kQSets, 2, z), 1024, dense_q_smem(Kmax), st>>>(d_tasks);
    launches_add(4);
    return cudaGetLastError();
}
template cudaError_t launch_stats_multi<float>(const StatsTask<float>*, const StatsTask<float>*, int, cudaStream_t);
template cudaError_t launch_stats_multi<double>(const StatsTask<double>*, const StatsTask<double>*, int, cudaStream_t);

template <class T>
cudaError_t launch_stats(const T* es, int K, int64_t P, T* stats, void* scratch, cudaStream_t st) {
    if (K <= 0 || P <= 0) return cudaSuccess;
    return launch_stats_ragged<T>(es, K, P, nullptr, P, stats, scratch, st);
}
template cudaError_t launch_stats<float>(const float*, int, int64_t, float*, void*, cudaStream_t);
template cudaError_t launch_stats<double>(const double*, int, int64_t, double*, void*, cudaStream_t);

}  // namespace gsea
