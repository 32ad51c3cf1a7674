// k_sort_bucket.cu -- per-permutation stable ranking of genes by metric: a
// one-pass bucket sort in shared memory (the order, ranks and weights of
// k_sort.cu's radix sorts, which take the permutations it declines).
//
// A radix sort moves every key once per digit and spends its time ranking
// equal digits (one ballot per bit: 63 us for one permutation of 20,000 fp32
// genes on an SM, ALU bound).  Metric values are spread over a continuous
// range, so one pass into about as many buckets as there are genes leaves one
// or two keys per bucket, and the rest is a handful of compares:
//   1. a coarse histogram of the top bits of the 32-bit radix image (sign,
//      exponent, one or two mantissa bits: a half or quarter octave per bin),
//      over a quarter of the keys, gives each bin as many buckets as it holds
//      keys; inside a bin the remaining bits interpolate linearly.  The map
//      key -> bucket never decreases, whatever the histogram, so only the
//      bucket sizes depend on the sampling.  The quarter is eight genes of
//      every 32, so that it does not depend on how the table orders its genes
//      (sampled(); one row of threads in four saw none of the wide genes of a
//      table ordered by scale, and every permutation of it was declined: 1,000
//      of 20,000 genes ordered so 539 -> 208 us);
//   2. the keys of every bucket are counted (16-bit counters, two to a word)
//      and the counts scanned;
//   3. (key, gene) pairs go to their bucket's slots in any order;
//   4. a pair's rank is its bucket's start plus the number of pairs of the
//      bucket that order before it (smaller key, or an equal key of a lower
//      gene: the stable order).
// Buckets of more than kBig pairs are ties in practice (constant or absent
// genes give one common key): if all their keys are equal they are ranked by
// gene through a bitmap, without compares.  A permutation with a large bucket
// of distinct keys, more tie buckets than pay (max_ties), or too many compares in all
// is marked in hard[] and left to the radix sort launched after this kernel.
//
// Keys crowded into a few values (counts under a difference of means) are left
// too, and found early: the counters of step 2 are fought over there, and a
// class mean's rounding makes neighbouring floats of one value, so that
// their buckets are large and distinct.  Threads compare keys of their own;
// with more than a dozen equal pairs (zeros, infinities and NaN apart), which
// stand for some 50 genes to a value whatever the number of genes, step 2 is
// not begun, and after two such permutations in a row a CTA looks at every
// fourth only.  Radix sort alone, found at the end, found early (counts, 60
// samples): 1,000 permutations of 20,000 genes 395, 480, 418 us; 2,000 of 3,000 200,
// 253, 218; 400 of 40,000 510, 562, 522; ten groups of 300 equal genes among 20,000
// 415, 752, 435.
//
// fp64 keys: the 32-bit image is the key rounded down to a float-like
// pattern (11-bit exponent clamped to 8 bits, 23 mantissa bits), which never
// decreases; pairs whose images tie are compared by their full keys.
//
// Shapes: up to 20,480 genes a thread keeps its keys in registers (ITEMS per
// thread) and the whole permutation has slots; 256 / 512 / 1,024 threads, so
// that small permutations share an SM.  Beyond (to 65,535 genes) the bucket
// counters of all genes stay in shared memory and the slots are filled and
// ranked one window of buckets after the other, the keys read again (from
// L2) for each window.
//
// Measured (GB300, the sort stage, radix sorts before -> this): 1,000
// permutations of 20,000 genes fp32 417 -> 197 us, fp64 1,724 -> 346 us; 300 x
// 60,000 fp32 713 -> 287 us; 1,024 x 2,000 fp32 105 -> 32 us.  Issue slots and
// the latency of shared memory between the barriers bound it (22 M warp
// instructions per 152 permutations of 20,000 genes at 62% issue activity;
// DRAM traffic is the keys once).
#include "common.cuh"
#include "kernels.h"

namespace gsea {
namespace {

constexpr int kBig = 64;        // pairs of a bucket ranked by compares
// tie buckets of a permutation that are still faster than the radix sort: one
// takes 9 us of 1,000 permutations of 1,000 genes (where the radix sort takes
// 194), 20 at 3,000 (200), 65 at 7,000 (250), 75 to 150 at 20,000 (395), 50 to 150 of
// 300 at 60,000 (690)
template <int NT, int ITEMS>
constexpr int max_ties() { return NT == 256 ? 16 : ITEMS == 20 ? 2 : 4; }
constexpr int kMaxCompares = 16;  // compares per gene on average
constexpr int kMaxWindows = 16;
constexpr int kSample = 4;      // one key in four enters the coarse histogram (beyond one row of threads)

template <int NT>
constexpr int coarse_bits() { return NT >= 1024 ? 11 : 10; }

// 32-bit image of a key, ascending in the output order (never decreasing in
// the key; exact for fp32)
__device__ __forceinline__ uint32_t image32(float v, bool descending) { return RadixKey<float>::from(v, descending); }
__device__ __forceinline__ uint32_t image32(double v, bool descending) {
    const unsigned long long bits = bits_of(v);
    const uint32_t hi = (uint32_t)(bits >> 32) & 0x7fffffffu, lo = (uint32_t)bits;
    uint32_t mag;
    if (hi < (896u << 20)) mag = 0u;                       // below float's normal range
    else if (hi >= (1151u << 20)) mag = 0x7f800000u;       // above it, infinity, NaN
    else mag = ((hi - (896u << 20)) << 3) | (lo >> 29);
    const uint32_t u = (bits >> 63) ? ~mag & 0x7fffffffu : mag | 0x80000000u;
    return descending ? ~u : u;
}

// The keys of the coarse histogram: gene g = i * NT + t (row i of the block's
// threads) with (t / 8) % kSample == i % kSample -- a sector of 32 bytes
// of each 128 in fp32, so that a pass over them loads no more than it uses, and
// another one in the next row.  Up to NT genes all of them.
__host__ __device__ __forceinline__ int sampled_row(int t) { return (t >> 3) & (kSample - 1); }
// buckets of a permutation: kSample times the sampled keys (16-bit indices)
__host__ __device__ __forceinline__ int bucket_count(int G, int NT) {
    if (G <= NT) return G;
    const int rows = G / NT, rest = G - rows * NT;
    int last = (rest & 31) - 8 * (rows & (kSample - 1));  // of the last, partial row
    last = last < 0 ? 0 : last > 8 ? 8 : last;
    const int n = kSample * (rows * (NT / kSample) + 8 * (rest >> 5) + last);
    return n < 65534 ? n : 65534;
}

struct Layout {
    uint32_t c, key, gene, rank, bitmap, bytes;  // byte offsets behind the coarse bins
    __host__ __device__ Layout(int G, int NB, int cap, bool stage_ranks, int coarse) {
        uint32_t o = 8u << coarse;
        c = o;
        o += 4u * (uint32_t)((NB >> 1) + 1);
        key = o;
        o += 4u * (uint32_t)cap;
        bitmap = o;
        o += 4u * (uint32_t)((G + 31) >> 5);
        gene = o;
        o += 2u * (uint32_t)((cap + 1) & ~1);
        o = (o + 3u) & ~3u;
        rank = o;
        if (stage_ranks) o += 2u * (uint32_t)((G + 1) & ~1);
        bytes = (o + 15u) & ~15u;
    }
};

// exclusive prefix of v over the block (one barrier; `sums` is written before
// it and read after it, so a caller passes an array no other phase uses)
template <int NT>
__device__ __forceinline__ uint32_t block_exclusive(uint32_t v, uint32_t* sums, uint32_t& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) sums[warp] = incl;
    __syncthreads();
    const uint32_t w = lane < NT / 32 ? sums[lane] : 0u;
    uint32_t wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFullMask, wi, o);
        if (lane >= o) wi += y;
    }
    total = __shfl_sync(kFullMask, wi, 31);
    return __shfl_sync(kFullMask, wi - w, warp) + incl - v;
}

struct BigBucket {
    uint32_t b, n, start;  // bucket, pairs, first slot of the buckets after it
};

template <class T, int NT, int ITEMS>
__device__ __forceinline__ void
sort_bucket_body(int bx, int gx, const T* __restrict__ keys, int G, int num_perms, bool descending, uint16_t* ranks,
                 T* __restrict__ sorted_abs, uint32_t* __restrict__ order, uint8_t* __restrict__ hard, int cap) {
    constexpr bool REGS = ITEMS > 0;       // keys in registers, every pair has a slot
    constexpr int CB = coarse_bits<NT>();
    constexpr int NC = 1 << CB;
    constexpr int BPT = NC / NT;           // coarse bins per thread
    static_assert(NC % NT == 0, "whole coarse bins per thread");
    static_assert(ITEMS % kSample == 0 && NT % 32 == 0, "sampled rows");
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t s_scan[3][32];
    constexpr int kMaxBig = max_ties<NT, ITEMS>();
    __shared__ BigBucket s_big[kMaxBig];
    __shared__ uint32_t s_nbig, s_pairs, s_bad, s_first, s_alike;
    __shared__ uint32_t s_wb[kMaxWindows + 1], s_wp[kMaxWindows + 1];  // windows: first bucket, first slot

    const int tid = threadIdx.x;
    const int NB = bucket_count(G, NT);
    const Layout L(G, NB, cap, REGS, CB);
    uint2* const H = reinterpret_cast<uint2*>(smem);  // coarse bin: first bucket, buckets
    uint32_t* const C = reinterpret_cast<uint32_t*>(smem + L.c);  // bucket counters, two 16-bit halves a word
    const uint16_t* const Ch = reinterpret_cast<const uint16_t*>(C);
    uint32_t* const skey = reinterpret_cast<uint32_t*>(smem + L.key);
    uint16_t* const sgene = reinterpret_cast<uint16_t*>(smem + L.gene);
    uint16_t* const srank = reinterpret_cast<uint16_t*>(smem + L.rank);  // REGS only
    uint32_t* const bitmap = reinterpret_cast<uint32_t*>(smem + L.bitmap);
    const int CW = (NB >> 1) + 1, BW = (G + 31) >> 5;
    const int wpt = ((CW + NT - 1) / NT) | 1;  // counter words per thread (odd: no bank conflicts)

    auto bucket_of = [&](uint32_t a) -> uint32_t {
        const uint2 h = H[a >> (32 - CB)];
        const uint32_t b = h.x + __umulhi(a << CB, h.y);
        return b < (uint32_t)NB ? b : (uint32_t)NB - 1u;
    };
    // images a table may have many of without being crowded: constant and absent
    // genes have 0 or NaN, those absent from one class an infinity in the ratios
    auto common = [&](uint32_t k) {
        const uint32_t u = descending ? ~k : k;
        return u == 0x80000000u || u == 0x7fffffffu || u == 0xffffffffu || u == 0xff800000u || u == 0x007fffffu;
    };
    constexpr int NREG = REGS ? ITEMS : 1;
    constexpr bool AHEAD = REGS && sizeof(T) == 4;  // the next permutation's keys are loaded early
    T ahead[AHEAD ? NREG : 1];
    bool loaded = false;  // the keys of the permutation at hand
    for (int w = tid; w < BW; w += NT) bitmap[w] = 0u;

    int left = 0;  // permutations left in a row
    for (int p = bx; p < num_perms; p += gx) {
        // crowded keys are a matter of the table, not of the permutation: after
        // two in a row only every fourth is looked at
        if (left >= 2 && (left & 3) != 0) {
            if (tid == 0) hard[p] = 1;
            left++;
            continue;
        }
        const T* const kp = keys + (int64_t)p * G;
        const int64_t base = (int64_t)p * G;
        uint32_t a[NREG];
        if constexpr (AHEAD) {
            if (!loaded) {
#pragma unroll
                for (int i = 0; i < NREG; i++) {
                    const int g = tid + i * NT;
                    ahead[i] = g < G ? kp[g] : T(0);
                }
            }
            loaded = false;
        }
        if constexpr (REGS) {
#pragma unroll
            for (int i = 0; i < NREG; i++) {
                const int g = tid + i * NT;
                if constexpr (AHEAD) a[i] = image32(ahead[i], descending);
                else a[i] = g < G ? image32(kp[g], descending) : 0u;
            }
        }
        // f(image, gene) for every gene of the thread
        auto each = [&](auto&& f) {
            if constexpr (REGS) {
#pragma unroll
                for (int i = 0; i < NREG; i++) {
                    const int g = tid + i * NT;
                    if (g < G) f(a[i], g);
                }
            } else {
                constexpr int U = 4;  // loads in flight
                for (int g0 = tid; g0 < G; g0 += U * NT) {
                    T v[U];
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const int g = g0 + u * NT;
                        v[u] = g < G ? kp[g] : T(0);
                    }
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const int g = g0 + u * NT;
                        if (g < G) f(image32(v[u], descending), g);
                    }
                }
            }
        };

        // 1. coarse histogram -> first bucket and number of buckets per bin
#pragma unroll
        for (int j = 0; j < BPT; j++) H[tid + j * NT].y = 0u;
        for (int w = tid; w < CW; w += NT) C[w] = 0u;
        if (tid == 0) s_nbig = s_pairs = s_bad = s_alike = 0u;
        __syncthreads();
        {
            const int row = sampled_row(tid);
            if constexpr (REGS) {
                if (G <= NT) {
                    if (tid < G) atomicAdd(&H[a[0] >> (32 - CB)].y, 1u);
                } else {
#pragma unroll
                    for (int i = 0; i < NREG; i += kSample) {
                        const uint32_t k01 = row & 1 ? a[i + 1] : a[i], k23 = row & 1 ? a[i + 3] : a[i + 2];
                        if (tid + (i + row) * NT < G)
                            atomicAdd(&H[(row & 2 ? k23 : k01) >> (32 - CB)].y, (uint32_t)kSample);
                    }
                }
            } else {
                constexpr int U = 4;  // loads in flight
                for (int g0 = tid + row * NT; g0 < G; g0 += U * kSample * NT) {
                    T v[U];
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const int g = g0 + u * kSample * NT;
                        v[u] = g < G ? kp[g] : T(0);
                    }
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        if (g0 + u * kSample * NT < G)
                            atomicAdd(&H[image32(v[u], descending) >> (32 - CB)].y, (uint32_t)kSample);
                    }
                    bool alike = false;
#pragma unroll
                    for (int u = 0; u < U; u += 2) {
                        const uint32_t k = image32(v[u], descending);
                        alike |= g0 + (u + 1) * kSample * NT < G && k == image32(v[u + 1], descending) && !common(k);
                    }
                    if (alike) atomicAdd(&s_alike, 1u);
                }
            }
        }
        __syncthreads();
        {
            uint32_t c[BPT], sum = 0, total;
#pragma unroll
            for (int j = 0; j < BPT; j++) {
                c[j] = H[tid * BPT + j].y;
                sum += c[j];
            }
            // here the block waits for the scan; up to 2,048 genes the rest costs
            // no more than the look (15 us of 2,000 permutations of 1,000)
            if constexpr (REGS && NT > 256) {
                bool alike = false;
#pragma unroll
                for (int i = 0; i < NREG; i += 4) alike |= a[i] == a[i + 1];
                if (__any_sync(kFullMask, alike)) {
                    alike = false;
#pragma unroll
                    for (int i = 0; i < NREG; i += 4)
                        alike |= tid + (i + 1) * NT < G && a[i] == a[i + 1] && !common(a[i]);
                    if (alike) atomicAdd(&s_alike, 1u);
                }
            }
            uint32_t run = block_exclusive<NT>(sum, s_scan[0], total);
#pragma unroll
            for (int j = 0; j < BPT; j++) {
                H[tid * BPT + j].x = run;
                run += c[j];
            }
        }
        __syncthreads();
        if (s_alike > (REGS ? 12u : 8u)) {  // crowded keys; of G / 4 or G / 8 pairs (uniform)
            if (tid == 0) hard[p] = 1;
            left++;
            __syncthreads();  // the flags are cleared next
            continue;
        }
        // 2. pairs per bucket, scanned.  With the keys in registers a pair
        // keeps its bucket and the count before it (its place in the bucket)
        // and C becomes the buckets' first slots; else one past their last
        uint32_t place[NREG];
        if constexpr (REGS) {
#pragma unroll
            for (int i = 0; i < NREG; i++) {
                place[i] = 0u;
                if (tid + i * NT < G) {
                    const uint32_t b = bucket_of(a[i]), sh = (b & 1u) << 4;
                    const uint32_t before = atomicAdd(&C[b >> 1], 1u << sh) >> sh;
                    place[i] = b | (before << 16);
                }
            }
        } else {
            each([&](uint32_t k, int) {
                const uint32_t b = bucket_of(k);
                atomicAdd(&C[b >> 1], 1u << ((b & 1u) << 4));
            });
        }
        __syncthreads();
        uint32_t slots;  // pairs with a slot: those of buckets ranked by compares
        {
            uint32_t sum = 0, pairs = 0;
            for (int j = 0; j < wpt; j++) {
                const int w = tid * wpt + j;
                if (w >= CW) break;
                uint32_t v = C[w];
                const uint32_t c0 = v & 0xffffu, c1 = v >> 16;
                if (max(c0, c1) > (uint32_t)kBig) {
                    for (int h = 0; h < 2; h++) {
                        const uint32_t n = h ? c1 : c0;
                        if (n <= (uint32_t)kBig) continue;
                        const uint32_t at = atomicAdd(&s_nbig, 1u);
                        if (at < (uint32_t)kMaxBig) s_big[at] = BigBucket{(uint32_t)(2 * w + h), n, 0u};
                        v &= h ? 0x0000ffffu : 0xffff0000u;
                    }
                    C[w] = v;
                }
                const uint32_t d0 = v & 0xffffu, d1 = v >> 16;
                sum += d0 + d1;
                pairs += d0 * d0 + d1 * d1;
            }
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) pairs += __shfl_xor_sync(kFullMask, pairs, o);
            if ((tid & 31) == 0) atomicAdd(&s_pairs, pairs);
            uint32_t run = block_exclusive<NT>(sum, s_scan[1], slots);
            for (int j = 0; j < wpt; j++) {
                const int w = tid * wpt + j;
                if (w >= CW) break;
                const uint32_t v = C[w];
                const uint32_t s1 = run + (v & 0xffffu), e1 = s1 + (v >> 16);
                C[w] = REGS ? run | (s1 << 16) : s1 | (e1 << 16);
                run = e1;
            }
        }
        __syncthreads();
        const int nbig = (int)min(s_nbig, (uint32_t)kMaxBig + 1u);
        const int W = cap - kBig;  // slots a window starts buckets in
        const int windows = REGS ? 1 : (int)((slots + W - 1) / W);
        bool give_up = nbig > kMaxBig || s_pairs > (uint32_t)kMaxCompares * (uint32_t)G + (uint32_t)kBig * kBig ||
                       windows > kMaxWindows;
        if (!REGS && !give_up) {
            if (tid <= windows) {  // first bucket that starts at or after slot tid * W
                uint32_t lo = 0, hi = (uint32_t)NB;
                const uint32_t want = (uint32_t)(tid * W);
                if (tid == windows) lo = hi;
                while (lo < hi) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if ((mid ? (uint32_t)Ch[mid - 1] : 0u) >= want) hi = mid; else lo = mid + 1;
                }
                s_wb[tid] = lo;
                s_wp[tid] = tid == windows ? slots : (lo ? (uint32_t)Ch[lo - 1] : 0u);
            }
        }
        if (nbig > 0 && !give_up) {
            // ties: where their ranks start (the slots of the buckets before,
            // read before step 3 takes slots), then each in turn
            if (tid < nbig) {
                const uint32_t b = s_big[tid].b;
                uint32_t st = REGS ? (uint32_t)Ch[b] : b ? (uint32_t)Ch[b - 1] : 0u;
                for (int j = 0; j < nbig; j++)
                    if (s_big[j].b < b) st += s_big[j].n;
                s_big[tid].start = st;
            }
            for (int j = 0; j < nbig; j++) {
                __syncthreads();
                if (tid == 0) s_first = 0xffffffffu;
                __syncthreads();
                const uint32_t big = s_big[j].b;
                uint32_t mine = 0xffffffffu;
                each([&](uint32_t k, int g) {
                    if (bucket_of(k) == big) {
                        mine = min(mine, (uint32_t)g);
                        atomicOr(&bitmap[g >> 5], 1u << (g & 31));
                    }
                });
                if (mine != 0xffffffffu) atomicMin(&s_first, mine);
                __syncthreads();
                const T ref = kp[s_first];
                const typename RadixKey<T>::U kref = RadixKey<T>::from(ref, descending);
                bool differs = false;
                each([&](uint32_t k, int g) {
                    if (bucket_of(k) == big) differs |= RadixKey<T>::from(kp[g], descending) != kref;
                });
                if (differs) s_bad = 1u;
                __syncthreads();
                const bool bad = s_bad != 0u;
                const int per = (BW + NT - 1) / NT;
                uint32_t n = 0, total;
                for (int i = 0; i < per; i++) {
                    const int w = tid * per + i;
                    if (w < BW) n += __popc(bitmap[w]);
                }
                uint32_t r = s_big[j].start + block_exclusive<NT>(n, s_scan[2], total);
                for (int i = 0; i < per; i++) {
                    const int w = tid * per + i;
                    if (w >= BW) break;
                    uint32_t bits = bitmap[w];
                    bitmap[w] = 0u;
                    if (bad) continue;
                    while (bits) {
                        const uint32_t g = (uint32_t)(w << 5) + (uint32_t)__ffs(bits) - 1u;
                        bits &= bits - 1u;
                        if constexpr (REGS) srank[g] = (uint16_t)r;
                        else ranks[base + r] = (uint16_t)g;
                        sorted_abs[base + r] = cuabs(ref);
                        if (order) order[base + r] = g;
                        r++;
                    }
                }
                if (bad) break;  // uniform
            }
            __syncthreads();
            give_up = s_bad != 0u;
        }
        if (tid == 0) hard[p] = give_up ? 1 : 0;
        if (give_up) {
            left++;
            __syncthreads();  // the counters and flags are cleared next
            continue;
        }
        left = 0;
        if (!REGS) __syncthreads();  // the windows' bounds
        for (int win = 0; win < windows; win++) {
            const uint32_t b_lo = REGS ? 0u : s_wb[win], b_hi = REGS ? (uint32_t)NB : s_wb[win + 1];
            const uint32_t p_lo = REGS ? 0u : s_wp[win], p_hi = REGS ? slots : s_wp[win + 1];
            // 3. pairs to slots; afterwards C = the buckets' first slots
            auto is_big = [&](uint32_t b) {
                bool big = false;
                for (int j = 0; j < nbig; j++) big |= s_big[j].b == b;
                return big;
            };
            if constexpr (REGS) {
                auto put = [&](int i) {
                    const uint32_t slot = (uint32_t)Ch[place[i] & 0xffffu] + (place[i] >> 16);
                    skey[slot] = a[i];
                    sgene[slot] = (uint16_t)(tid + i * NT);
                };
                if (nbig == 0) {
#pragma unroll
                    for (int i = 0; i < NREG; i++)
                        if (tid + i * NT < G) put(i);
                } else {
#pragma unroll
                    for (int i = 0; i < NREG; i++)
                        if (tid + i * NT < G && !is_big(place[i] & 0xffffu)) put(i);
                }
            } else {
                each([&](uint32_t k, int g) {
                    const uint32_t b = bucket_of(k);
                    if (b < b_lo || b >= b_hi || is_big(b)) return;
                    const uint32_t sh = (b & 1u) << 4;
                    const uint32_t slot = ((atomicSub(&C[b >> 1], 1u << sh) >> sh) & 0xffffu) - 1u - p_lo;
                    skey[slot] = k;
                    sgene[slot] = (uint16_t)g;
                });
            }
            if constexpr (AHEAD) {
                const int pn = p + gx;
                loaded = pn < num_perms;
                if (loaded) {
#pragma unroll
                    for (int i = 0; i < NREG; i++) {
                        const int g = tid + i * NT;
                        ahead[i] = g < G ? keys[(int64_t)pn * G + g] : T(0);
                    }
                }
            }
            __syncthreads();
            // 4. ranks: the bucket's start plus the pairs before in it
            const int n = (int)(p_hi - p_lo);
            constexpr int U = 4;
            for (int i0 = tid; i0 < n; i0 += U * NT) {
                uint32_t k[U], s[U], e[U], r[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int i = i0 + u * NT;
                    k[u] = s[u] = e[u] = 0u;
                    if (i < n) {
                        k[u] = skey[i];
                        const uint32_t b = bucket_of(k[u]);
                        s[u] = (uint32_t)Ch[b] - p_lo;
                        e[u] = (!REGS && b + 1u == b_hi ? p_hi : (uint32_t)Ch[b + 1u]) - p_lo;
                    }
                    r[u] = s[u] + p_lo;
                }
                if (nbig > 0) {
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const uint32_t b = bucket_of(k[u]);
                        for (int j = 0; j < nbig; j++) r[u] += s_big[j].b < b ? s_big[j].n : 0u;
                    }
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int i = i0 + u * NT;
                    if (i >= n) break;
                    uint32_t same = 0u;
                    if (e[u] - s[u] > 1u) {
#pragma unroll 1
                        for (uint32_t j = s[u]; j < e[u]; j++) {
                            const uint32_t kj = skey[j];
                            r[u] += kj < k[u] ? 1u : 0u;
                            same += kj == k[u] ? 1u : 0u;
                        }
                    }
                    const uint32_t g = sgene[i];
                    T v;
                    if constexpr (sizeof(T) == 8) v = kp[g];
                    else {
                        uint32_t x = descending ? ~k[u] : k[u];
                        x = (x & 0x80000000u) ? (x & 0x7fffffffu) : ~x;
                        v = __uint_as_float(x);
                    }
                    if (same > 1u) {  // equal images: full keys, then genes
                        const typename RadixKey<T>::U kf = RadixKey<T>::from(v, descending);
#pragma unroll 1
                        for (uint32_t j = s[u]; j < e[u]; j++) {
                            if (skey[j] != k[u]) continue;
                            const uint32_t gj = sgene[j];
                            if constexpr (sizeof(T) == 8) {
                                const typename RadixKey<T>::U kj = RadixKey<T>::from(kp[gj], descending);
                                r[u] += (kj < kf || (kj == kf && gj < g)) ? 1u : 0u;
                            } else {
                                r[u] += gj < g ? 1u : 0u;
                            }
                        }
                    }
                    if constexpr (REGS) srank[g] = (uint16_t)r[u];
                    else ranks[base + r[u]] = (uint16_t)g;  // the order, until the last window is done
                    sorted_abs[base + r[u]] = cuabs(v);
                    if (order) order[base + r[u]] = g;
                }
            }
            __syncthreads();
        }
        if constexpr (REGS) {
            if ((base & 1) == 0) {  // two ranks a store
                uint32_t* const r2 = reinterpret_cast<uint32_t*>(ranks + base);
                const uint32_t* const s2 = reinterpret_cast<const uint32_t*>(srank);
                for (int w = tid; w < G >> 1; w += NT) r2[w] = s2[w];
                if ((G & 1) && tid == 0) ranks[base + G - 1] = srank[G - 1];
            } else {
                for (int g = tid; g < G; g += NT) ranks[base + g] = srank[g];
            }
        } else {
            // the order becomes ranks by gene, turned round in shared memory
            uint16_t* const sr = reinterpret_cast<uint16_t*>(smem);
            for (int i = tid; i < G; i += NT) sr[ranks[base + i]] = (uint16_t)i;
            __syncthreads();
            for (int g = tid; g < G; g += NT) ranks[base + g] = sr[g];
            __syncthreads();
            for (int w = tid; w < BW; w += NT) bitmap[w] = 0u;
        }
    }
}

template <int NT>
constexpr int min_blocks() { return NT >= 1024 ? 1 : NT == 512 ? 2 : 5; }

template <class T, int NT, int ITEMS>
__global__ void __launch_bounds__(NT, min_blocks<NT>())
sort_bucket_kernel(const T* __restrict__ keys, int G, int num_perms, bool descending, uint16_t* ranks,
                   T* __restrict__ sorted_abs, uint32_t* __restrict__ order, uint8_t* __restrict__ hard, int cap) {
    sort_bucket_body<T, NT, ITEMS>(blockIdx.x, gridDim.x, keys, G, num_perms, descending, ranks, sorted_abs, order,
                                   hard, cap);
}

constexpr int kSmemCap = 232448 - 1024;  // a CTA's shared memory, less the static part

// slots of a window of the form without registers: what the bucket counters
// and the bitmap leave (the ranks by gene are turned round over all of it)
template <int NT>
int window_cap(int G) {
    const int left = kSmemCap - (int)Layout(G, bucket_count(G, NT), 0, false, coarse_bits<NT>()).bytes - 16;
    const int cap = left / 6;
    return cap < G + kBig ? cap : G + kBig;
}

// every instance of a batch of one shape: blockIdx.z = the instance
template <class T, int NT, int ITEMS>
__global__ void __launch_bounds__(NT, min_blocks<NT>()) sort_bucket_multi(const SortTask* __restrict__ tasks) {
    const SortTask t = tasks[blockIdx.z];
    sort_bucket_body<T, NT, ITEMS>(blockIdx.x, gridDim.x, static_cast<const T*>(t.keys), t.G, t.num_perms,
                                   t.descending != 0, static_cast<uint16_t*>(t.ranks), static_cast<T*>(t.sorted),
                                   t.order, t.hard, t.cap);
}

template <class T, int NT, int ITEMS>
size_t bucket_smem(int G, int cap) {
    return Layout(G, bucket_count(G, NT), cap, ITEMS > 0, coarse_bits<NT>()).bytes;
}

int sm_count() {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
}

template <class T, int NT, int ITEMS>
cudaError_t launch_bucket(const T* keys, int G, int P, bool desc, const SortBuffers& o, cudaStream_t st) {
    const int cap = ITEMS > 0 ? G : window_cap<NT>(G);
    const size_t smem = bucket_smem<T, NT, ITEMS>(G, cap);
    auto kern = sort_bucket_kernel<T, NT, ITEMS>;
    cudaError_t e = allow_smem(kern, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, NT, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidValue;
    const int fill = sm_count() * per_sm;
    kern<<<P < fill ? P : fill, NT, smem, st>>>(keys, G, P, desc, static_cast<uint16_t*>(o.ranks),
                                                static_cast<T*>(o.sorted_abs), o.order, o.hard, cap);
    launches_add(1);
    return cudaGetLastError();
}

template <class T, int NT, int ITEMS>
cudaError_t launch_bucket_multi(const SortTask* d, const SortTask* h, int n, cudaStream_t st) {
    size_t smem = 0;
    for (int i = 0; i < n; i++) {
        const size_t s = bucket_smem<T, NT, ITEMS>(h[i].G, h[i].cap);
        smem = s > smem ? s : smem;
    }
    auto kern = sort_bucket_multi<T, NT, ITEMS>;
    cudaError_t e = allow_smem(kern, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, NT, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidValue;
    const int per = (2 * sm_count() * per_sm + n - 1) / n;  // CTAs per instance: about two waves in all
    kern<<<dim3((unsigned)(per > 0 ? per : 1), 1, (unsigned)n), NT, smem, st>>>(d);
    launches_add(1);
    return cudaGetLastError();
}

}  // namespace

// threads and keys per thread by the number of genes (0: no bucket form);
// keyed threads * 100 + items
int sort_bucket_class(int G) {
    if (G < 1 || G > 65535) return 0;
    if (G <= 256 * 8) return 25608;
    if (G <= 512 * 8) return 51208;
    if (G <= 512 * 20) return 51220;
    if (G <= 1024 * 20) return 102420;
    return 102400;
}
// a batch launches each class it has instances of: fewer classes
int sort_bucket_multi_class(int G) {
    const int c = sort_bucket_class(G);
    return c == 51208 ? 51220 : c;
}
int sort_bucket_cap(int G) { return G <= 1024 * 20 ? G : window_cap<1024>(G); }

template <class T>
cudaError_t launch_sort_bucket(const T* keys, int G, int P, bool descending, const SortBuffers& o, cudaStream_t st) {
    switch (sort_bucket_class(G)) {
        case 25608: return launch_bucket<T, 256, 8>(keys, G, P, descending, o, st);
        case 51208: return launch_bucket<T, 512, 8>(keys, G, P, descending, o, st);
        case 51220: return launch_bucket<T, 512, 20>(keys, G, P, descending, o, st);
        case 102420: return launch_bucket<T, 1024, 20>(keys, G, P, descending, o, st);
        case 102400: return launch_bucket<T, 1024, 0>(keys, G, P, descending, o, st);
        default: return cudaErrorInvalidValue;
    }
}
template cudaError_t launch_sort_bucket<float>(const float*, int, int, bool, const SortBuffers&, cudaStream_t);
template cudaError_t launch_sort_bucket<double>(const double*, int, int, bool, const SortBuffers&, cudaStream_t);

template <class T>
static cudaError_t bucket_multi(const SortTask* d, const SortTask* h, int n, int cls, cudaStream_t st) {
    switch (cls) {
        case 25608: return launch_bucket_multi<T, 256, 8>(d, h, n, st);
        case 51220: return launch_bucket_multi<T, 512, 20>(d, h, n, st);
        case 102420: return launch_bucket_multi<T, 1024, 20>(d, h, n, st);
        case 102400: return launch_bucket_multi<T, 1024, 0>(d, h, n, st);
        default: return cudaErrorInvalidValue;
    }
}
cudaError_t launch_sort_bucket_multi(const SortTask* d_tasks, const SortTask* h_tasks, int n, int cls, bool fp64,
                                     cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    if (n > 65535) return cudaErrorInvalidValue;
    return fp64 ? bucket_multi<double>(d_tasks, h_tasks, n, cls, st) : bucket_multi<float>(d_tasks, h_tasks, n, cls, st);
}

}  // namespace gsea
