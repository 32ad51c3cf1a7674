"""Tables whose keys crowd into a few values: the bucket sort leaves them to the
radix sort early enough to cost little more than the radix sort alone, and a
run of permutations it takes and leaves in turn is sorted right."""
import numpy as np
import pytest

from cudagsea_gb300 import synthetic
from cudagsea_gb300 import _native as N
from tests.test_parity_gpu import check_sort, run_plan

pytestmark = pytest.mark.gpu


def grouped(G, perms, groups, size, S=60):
    """`groups` groups of `size` genes with one row of values each."""
    d = synthetic.make(G, S, 2, perms, seed=5, n_class_b=S // 2, set_max=min(60, G))
    at = np.random.RandomState(1).permutation(G)
    for j in range(groups):
        d.exprs[:, at[j * size:(j + 1) * size]] = d.exprs[:, [at[j * size]]]
    return d


def counts(G, perms):
    d = synthetic.make(G, 60, 2, perms, seed=6, n_class_b=30, set_max=60)
    rs = np.random.RandomState(2)
    d.exprs = np.ascontiguousarray(rs.poisson(rs.lognormal(0.0, 1.5, G), (60, G)).astype(np.float32))
    return d


def sort_us(d, metric, double, variant):
    r = run_plan(d, metric, double=double, debug=False, tuning=dict(sort_variant=variant))
    p = r["plan"]
    p.set_profiling(True)
    ts = []
    for _ in range(9):
        p.execute()
        ts.append(p.stage_times()["sort"])
    p.close()
    return min(ts) * 1e3


@pytest.mark.parametrize("double", [False, True], ids=["f32", "f64"])
@pytest.mark.parametrize("kind", ["groups", "ratio", "counts"])
def test_crowded_tables_cost_little_more_than_the_radix_sort(gpu, kind, double):
    G, perms = 20000, 600
    metric = "naive_diff_of_classes"
    if kind == "groups":
        d = grouped(G, perms, 10, 300)
    elif kind == "ratio":  # half of the genes constant: their ratio is 1
        d = grouped(G, perms, 0, 0)
        d.exprs[:, ::2] = 5.0
        metric = "naive_ratio_of_classes"
    else:
        d = counts(G, perms)
    alone, behind = sort_us(d, metric, double, 3), sort_us(d, metric, double, 0)
    # found at the end: 1.8, 1.7 and 1.2 times the radix sort alone; a tenth is
    # the loads and the coarse histogram
    assert behind < 1.35 * alone, (behind, alone)


@pytest.mark.parametrize("double", [False, True], ids=["f32", "f64"])
@pytest.mark.parametrize("G,perms,groups,size", [(1000, 1300, 8, 62), (2500, 900, 6, 70), (22000, 330, 3, 90)])
def test_taken_and_left_in_turn(gpu, double, G, perms, groups, size):
    d = grouped(G, perms, groups, size)
    r = run_plan(d, "naive_diff_of_classes", double=double)
    left = r["plan"].read_buffer(N.BUF_SORT_LEFT, np.uint8, (perms,))
    assert left.any()
    check_sort(r["keys"], r["order"], r["ranks"], r["sorted"])
    r["plan"].close()
