"""Statistics of few permutations: the null histograms at the number of columns
where their threads change from scores to rows, bit for bit the oracle's, and
two permutations no slower than a hundred."""
import numpy as np
import pytest

import oracle
from cudagsea_gb300 import api
from tests.test_stats_steps_gpu import assert_same, device_stats, scores

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,P", [(3, 512), (3, 513), (3, 514), (3, 1025), (40, 513), (40, 514), (6142, 3),
                                 (14500, 2), (14500, 34), (14500, 256), (14500, 257), (33000, 2), (33000, 35)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64], ids=["f32", "f64"])
def test_columns_where_the_histogram_changes(gpu, K, P, dtype):
    if dtype == np.float64 and K > 14500:
        K = 15001  # the oracle's order of the observed scores grows with K^2
    es = scores(K, P, dtype)
    assert_same(device_stats(es), oracle.stats(es), K)


def stats_us(K, P):
    rs = np.random.RandomState(0)
    lab = np.r_[np.zeros(6), np.ones(6)].astype(np.uint8)
    x = (8 + rs.standard_normal((12, 64))).astype(np.float32)
    genes = np.argsort(rs.rand(K, 64), 1)[:, :5].astype(np.int32).ravel()
    p = api.Plan(64, 12, K, P, "naive_diff_of_classes")
    p.set_inputs(x, lab, np.arange(K + 1) * 5, genes)
    p.set_profiling(True)
    ts = []
    for _ in range(15):
        p.execute()
        ts.append(p.stage_times()["stats"])
    p.close()
    return float(np.sort(ts)[:8].mean()) * 1e3


def test_two_permutations_are_no_slower_than_a_hundred(gpu):
    few, many = stats_us(1000, 2), stats_us(1000, 100)
    # ten times as long a row of the matrix at a time
    assert few < 1.5 * many, (few, many)
