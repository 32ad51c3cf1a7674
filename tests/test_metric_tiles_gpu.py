"""The plain metric kernels at the edges of their tiles (32 to 128 genes, four
permutations a warp, 32 samples a copy, one to eight warps a block): keys
equal the oracle's bit for bit (log2 metrics: 2 ulp, the device's logarithm),
with 4 and 8 permutations a warp, rows on and off 16-byte boundaries, and
values that are not finite."""
import numpy as np
import pytest

import oracle
from cudagsea_gb300 import api, synthetic
from tests import helpers as H
from tests.test_parity_gpu import run_plan

pytestmark = pytest.mark.gpu

SHAPES = [(1, 2, 1), (31, 31, 3), (33, 33, 5), (127, 64, 4), (129, 65, 9), (260, 20, 33), (1028, 7, 130), (515, 200, 70)]


def check(metric, mine, ref):
    if metric in H.LOG_METRICS:
        bad = ~((H.ulp_diff(mine, ref) <= 2) | (np.isnan(mine) & np.isnan(ref)))
        assert not bad.any()
    else:
        u = np.uint64 if mine.dtype == np.float64 else np.uint32
        both = np.isnan(mine) & np.isnan(ref)
        assert np.array_equal(np.where(both, 0, mine.view(u)), np.where(both, 0, ref.view(u)))


@pytest.mark.parametrize("metric", range(14), ids=api.METRICS)
@pytest.mark.parametrize("double", [False, True], ids=["f32", "f64"])
def test_metric_keys_at_tile_edges(gpu, metric, double):
    for i, (G, S, P) in enumerate(SHAPES):
        d = synthetic.make(G, S, 2, P, seed=G + S, n_class_b=max(1, S // 3), set_min=1, set_max=min(9, G), clamp=1e-3)
        r = run_plan(d, metric, double=double, tuning=dict(metric_pb=8 if i & 1 else 4))
        x = d.exprs.astype(np.float64) if double else d.exprs
        check(metric, r["keys"], oracle.metric(metric, x, d.labels, P, double=double))
        r["plan"].close()


@pytest.mark.parametrize("metric", [0, 1, 3, 6, 8, 10, 12], ids=lambda m: api.METRICS[m])
@pytest.mark.parametrize("double", [False, True], ids=["f32", "f64"])
def test_metric_keys_of_values_that_are_not_finite(gpu, metric, double):
    d = synthetic.make(150, 34, 2, 10, seed=5, n_class_b=15, set_min=1, set_max=9, clamp=1e-3)
    d.exprs[3, 10:20] = np.inf
    d.exprs[5, 15:30] = -np.inf
    d.exprs[9, 40:45] = np.nan
    d.exprs[:, 60:64] = np.float32(3e38)
    r = run_plan(d, metric, double=double)
    x = d.exprs.astype(np.float64) if double else d.exprs
    check(metric, r["keys"], oracle.metric(metric, x, d.labels, 10, double=double))
    r["plan"].close()
