"""The statistics in four steps (k_stats.cu, dense form) at the edges of their
blocks: a set to a warp (8 and 4 to a block), 128 columns and 16 sets to an
extrema block, the histogram's shares of 1,024 scores, 1,024 bins to a suffix
round, and the last collection that the dense form takes with the next one.
Bit for bit the oracle's, with ties, zeros, a set of zeros and NaN."""
import ctypes

import numpy as np
import pytest

import oracle
from cudagsea_gb300 import _native as N

pytestmark = pytest.mark.gpu


def device_stats(es):
    import torch
    K, P = es.shape
    precision = 64 if es.dtype == np.float64 else 32
    need = ctypes.c_size_t(0)
    N.check(N.lib().gsea_stats_scratch_bytes(K, P, precision, ctypes.byref(need)))
    scratch = torch.full(((need.value + 255) // 256 * 256,), 0xa5, dtype=torch.uint8, device="cuda")
    x = torch.from_numpy(es).cuda()
    out = torch.empty(5 * K, dtype=x.dtype, device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    for _ in range(2):  # the second call finds the first one's scratch
        N.check(N.lib().gsea_stats_device(ptr(x), K, P, precision, ptr(out), ptr(scratch), scratch.numel(), None))
    torch.cuda.synchronize()
    return out.cpu().numpy()


def scores(K, P, dtype):
    rng = np.random.RandomState(K * 7 + P)
    es = rng.uniform(-1, 1, (K, P)).astype(dtype)
    es[rng.uniform(size=es.shape) < 0.1] = 0.0
    es[rng.uniform(size=es.shape) < 0.2] = 0.25
    if K > 4:
        es[1] = 0.0             # no score at all: 1 / 0
        es[2] = es[3]           # equal observed scores and equal nulls
        es[K - 1, P // 2] = np.nan
    if K > 8:
        es[4] = np.abs(es[4]) + dtype(0.125)
        es[5, 0] = np.nan
    return es


def assert_same(got, want, K):
    u = np.uint64 if got.dtype == np.float64 else np.uint32
    same = (got.view(u) == want.view(u)) | (np.isnan(got) & np.isnan(want))
    assert same.all(), [(int(i) // K, int(i) % K, got[i], want[i]) for i in np.flatnonzero(~same)[:5]]


@pytest.mark.parametrize("K", [1, 3, 4, 5, 8, 9, 17, 1021, 1022, 1023, 2049, 6140, 6150])
@pytest.mark.parametrize("P", [1, 2, 31, 33, 128, 130, 1025])
@pytest.mark.parametrize("dtype", [np.float32, np.float64], ids=["f32", "f64"])
def test_statistics_at_block_edges(gpu, K, P, dtype):
    if K > 1000 and P > 130:
        P = 130 + K % 7
    es = scores(K, P, dtype)
    assert_same(device_stats(es), oracle.stats(es), K)


@pytest.mark.parametrize("K,P", [(1, 2), (2, 9000), (5, 8193), (303, 40), (305, 33), (1023, 9), (6150, 12),
                                 (15000, 3), (20000, 4), (30000, 3)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64], ids=["f32", "f64"])
def test_ragged_form_with_every_column(gpu, K, P, dtype):
    """The weighted histogram with weights of 1: keys and counters in shared
    memory, keys only or (the largest collections) neither; sets over blocks, columns over blocks."""
    import torch
    es = scores(K, P, dtype)
    x = torch.from_numpy(es).cuda()
    counts = torch.full((K,), P, dtype=torch.int64, device="cuda")
    out = torch.empty(5 * K, dtype=x.dtype, device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    N.check(N.lib().gsea_stats_ragged(ptr(x), K, P, ptr(counts), P, 64 if dtype == np.float64 else 32, ptr(out), None))
    torch.cuda.synchronize()
    assert_same(out.cpu().numpy(), oracle.stats(es), K)


@pytest.mark.parametrize("scale", [1e-30, 1.0, 1e30])
def test_histogram_slots_over_the_range(gpu, scale):
    """Observed keys crowded at one end, of one value, zero, and huge."""
    K, P = 700, 60
    rng = np.random.RandomState(3)
    es = (rng.standard_normal((K, P)) * scale).astype(np.float32)
    es[:300, 0] = np.float32(scale) * (1 + np.arange(300) * np.float32(2.0 ** -22))
    es[300:400, 0] = np.float32(-scale)
    es[400] = np.float32(scale)   # normalised to exactly 1
    es[401:403, 0] = 0.0
    es[403, 0] = np.float32(3e37) if scale < 1e10 else np.float32(3e38)
    assert_same(device_stats(es), oracle.stats(es), K)
