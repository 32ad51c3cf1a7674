"""Double scores that the walk in fp32 cannot decide: sets with NaN weights
(absent genes under the ratios and signal to noise) against the oracle's
running sum, and no slower than the sets of a table without them."""
import numpy as np
import pytest

import oracle
from cudagsea_gb300 import synthetic
from tests import helpers as H
from tests.test_parity_gpu import check_sort, run_plan

pytestmark = pytest.mark.gpu


def absent(G, perms, frac, K=20, S=14, seed=0):
    """A table with absent genes (zero everywhere): NaN keys, ranked first or last."""
    d = synthetic.make(G, S, K, perms, seed=G + seed, n_class_b=S // 2, set_min=1, set_max=min(300, G))
    rs = np.random.RandomState(G + seed)
    d.exprs = np.abs(d.exprs)
    d.exprs[:, rs.uniform(size=G) < frac] = 0.0
    return d


@pytest.mark.parametrize("metric", ["naive_ratio_of_classes", "naive_log2_ratio_of_classes", "twopass_signal2noise"])
@pytest.mark.parametrize("ascending", [False, True])
@pytest.mark.parametrize("double", [False, True], ids=["f32", "f64"])
def test_nan_weights(gpu, metric, ascending, double):
    for G, frac in ((40, 0.5), (1500, 0.01), (1500, 1.0), (20000, 0.02), (45000, 0.3)):
        d = absent(G, 6, frac)
        r = run_plan(d, metric, double=double, ascending=ascending)
        sk, order = check_sort(r["keys"], r["order"], r["ranks"], r["sorted"], ascending=ascending)
        es_o = oracle.es(sk, order, d.set_offsets, d.set_genes)
        w = r["sorted"]
        for k in range(d.num_sets):
            members = d.set_genes[d.set_offsets[k]:d.set_offsets[k + 1]]
            for p in range(6):
                total = w[p, r["ranks"][p, members]].sum()
                if np.isnan(total) or np.isfinite(total):  # infinite sums: as the running sum leaves them
                    assert H.es_close(r["es"][k, p], es_o[k, p], double), (G, k, p, r["es"][k, p], es_o[k, p])
        r["plan"].close()


def es_us(d):
    r = run_plan(d, "twopass_signal2noise", double=True, debug=False)
    p = r["plan"]
    p.set_profiling(True)
    ts = []
    for _ in range(9):
        p.execute()
        ts.append(p.stage_times()["es"])
    p.close()
    return min(ts) * 1e3


def test_nan_weights_cost_no_walk_in_double(gpu):
    plain, some = es_us(absent(20000, 304, 0.0, K=300)), es_us(absent(20000, 304, 0.05, K=300))
    # walked twice in double it took 2.9 times as long
    assert some < 1.5 * plain, (some, plain)


@pytest.mark.parametrize("G", [64, 400, 6000, 20000, 50000])
def test_leads_around_the_margin_of_the_search(gpu, G):
    """Members at equal steps and weights that fall slowly: the running sum is
    flat around its extremum, and the leads of neighbouring hits pass from far
    above to far below what the walk in fp32 can tell.  The wrong hit would show
    in the score, which is held to the tolerance of double sums."""
    for slope in (1e-1, 1e-2, 1e-3, 1e-4, 1e-5, 1e-6, 1e-7):
        sets = [np.arange(a, G, step) for step in (2, 3, 7) for a in (0, step - 1)]
        sets.append(np.r_[np.arange(0, G // 2, 3), np.arange(G // 2, G, 5)])
        d = synthetic.make(G, 2, 1, 3, seed=1, n_class_b=1, set_min=1, set_max=1)
        keys = 1.0 + slope * np.linspace(0.5, -0.5, G) * (1 + 0.01 * np.sin(np.arange(G)))
        x = np.zeros((2, G))
        x[d.labels == 0] = keys  # one sample a class: the metric is its value
        d.exprs = x
        d.set_offsets = np.r_[0, np.cumsum([s.size for s in sets])].astype(np.int64)
        d.set_genes = np.concatenate(sets).astype(np.int32)
        r = run_plan(d, "naive_diff_of_classes", double=True)
        sk, order = check_sort(r["keys"], r["order"], r["ranks"], r["sorted"])
        es_o = oracle.es(sk, order, d.set_offsets, d.set_genes)
        same = H.es_close(r["es"], es_o, True) | H.es_close(r["es"], -es_o, True) & (
            np.abs(es_o) < 1e-9)  # both signs where the score is a rounding error
        assert same.all(), (slope, r["es"][~same][:3], es_o[~same][:3])
        r["plan"].close()
