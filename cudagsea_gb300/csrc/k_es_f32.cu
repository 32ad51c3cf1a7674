// k_es_f32.cu -- the fp32 instantiations of the enrichment kernels (k_es.cuh).
#include "k_es.cuh"

namespace gsea {

int es_size_class(int G) { return es_wpl(G, G <= 65536); }

namespace {
// The sets' marking lists (EsSets): one warp per set writes its groups and
// finds duplicates and unknown ids in a bitmap of the genes, from which the
// list of a set that has any is written again.  A set's list
// starts at group floor(offset / 128) + k, which leaves every set room for
// its last, partial group without a scan over the sets.
constexpr int kListWarps = 4;
__global__ void __launch_bounds__(32 * kListWarps)
es_lists_kernel(const int64_t* __restrict__ off, const int32_t* __restrict__ genes, int K, int G,
                int2* __restrict__ rec, uint2* __restrict__ list) {
    extern __shared__ uint32_t seen[];  // [kListWarps][(G + 31) / 32]
    const int words = (G + 31) >> 5;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t* const bm = seen + warp * words;
    for (int w = lane; w < words; w += 32) bm[w] = 0u;
    const int k = blockIdx.x * kListWarps + warp;
    if (k >= K) return;  // the whole warp; no block barrier below
    __syncwarp();
    const int64_t a = off[k];
    const int64_t m = off[k + 1] - a;
    const int64_t first = a / 128 + k;
    bool bad = false;
    for (int64_t base = 0; base < m; base += 128) {
        uint32_t e[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int64_t idx = base + 32 * i + lane;
            e[i] = 0u;
            if (idx < m) {
                const int g = genes[a + idx];
                if (g < 0 || g >= G) {
                    bad = true;
                } else {
                    e[i] = (uint32_t)g;
                    const uint32_t bit = 1u << (g & 31);
                    if (atomicOr(&bm[g >> 5], bit) & bit) bad = true;
                }
            }
        }
        list[(first + base / 128) * 32 + lane] = make_uint2(e[0] | (e[1] << 16), e[2] | (e[3] << 16));
    }
    bad = __any_sync(kFullMask, bad);
    int n = (int)m;  // fewer than 2^31 members to a set
    if (bad) {  // its genes once, ascending (what stays behind them in the last group are valid ids)
        __syncwarp();
        uint16_t* const entries = reinterpret_cast<uint16_t*>(list + first * 32);
        n = 0;
        for (int w0 = 0; w0 < words; w0 += 32) {
            uint32_t bits = w0 + lane < words ? bm[w0 + lane] : 0u;
            const int c = __popc(bits);
            int incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(kFullMask, incl, o);
                if (lane >= o) incl += y;
            }
            for (int at = n + incl - c; bits; at++, bits &= bits - 1u)
                entries[(at >> 7) * 128 + (at & 31) * 4 + ((at >> 5) & 3)] =
                    (uint16_t)((w0 + lane) * 32 + __ffs(bits) - 1);
            n += __shfl_sync(kFullMask, incl, 31);
        }
    }
    if (lane == 0) rec[k] = make_int2(bad ? ~(int)first : (int)first, n);
}
}  // namespace

size_t es_list_bytes(int64_t K, int64_t nnz) { return ((size_t)(nnz / 128 + K) + 1) * 128 * sizeof(uint16_t); }

cudaError_t launch_es_lists(const int64_t* off, const int32_t* genes, int K, int G, int2* rec, uint2* list,
                            cudaStream_t st) {
    if (K <= 0) return cudaSuccess;
    if (G > 65536) return cudaErrorInvalidValue;
    const size_t smem = sizeof(uint32_t) * kListWarps * (size_t)((G + 31) / 32);
    es_lists_kernel<<<(K + kListWarps - 1) / kListWarps, 32 * kListWarps, smem, st>>>(off, genes, K, G, rec, list);
    launches_add(1);
    return cudaGetLastError();
}

template cudaError_t launch_es<float>(const void*, bool, const float*, int, int, const EsSets&, const int32_t*,
                                      const float*, int, float*, int64_t, int64_t, cudaStream_t, EsTuning, const int*);
template cudaError_t launch_es_batch<float>(const EsTask<float>*, const int64_t*, int, int64_t, unsigned long long*,
                                            int, int, EsTuning, cudaStream_t);
template cudaError_t launch_decay_table<float>(int, float*, cudaStream_t);

}  // namespace gsea
