"""Sets that list a gene more than once or an unknown id: the scores of the set
without them, and in double no slower (the marking lists hold every gene once)."""
import numpy as np
import pytest

from cudagsea_gb300 import synthetic
from tests import helpers as H
from tests.test_parity_gpu import run_plan

pytestmark = pytest.mark.gpu


def with_sets(d, sets):
    d.set_offsets = np.r_[0, np.cumsum([len(s) for s in sets])].astype(np.int64)
    d.set_genes = np.concatenate(sets).astype(np.int32) if sets else np.zeros(0, np.int32)
    return d


def table(G, perms):
    return synthetic.make(G, 14, 1, perms, seed=G, n_class_b=7, set_min=1, set_max=1)


# one gene, the last and first sizes of a bitmap word and of a lane's words, the largest with lists and beyond
@pytest.mark.parametrize("G", [1, 32, 33, 1024, 4097, 20000, 20481, 65536, 65537])
@pytest.mark.parametrize("double", [False, True], ids=["f32", "f64"])
def test_duplicates_and_unknown_ids_fall_away(gpu, G, double):
    rs = np.random.RandomState(G)
    # around the groups of 128 entries, the lanes of 32, nothing, everything
    clean = [np.sort(rs.choice(G, size=min(G, n), replace=False)) for n in (1, 2, 31, 32, 33, 127, 128, 129, 400)]
    clean += [np.arange(0), np.arange(min(G, 3000))]
    behind, mixed = [], []
    for s in clean:
        more = np.r_[s[:5], s[-3:], [-1, G, 2 ** 31 - 1, -2 ** 31]].astype(np.int64)
        behind.append(np.r_[s, more])
        mixed.append(rs.permutation(np.r_[s, s, more]))
    perms = 5 if G > 20000 else 20
    ref = run_plan(with_sets(table(G, perms), clean), "naive_diff_of_classes", double=double, debug=False)
    a = run_plan(with_sets(table(G, perms), behind), "naive_diff_of_classes", double=double, debug=False)
    b = run_plan(with_sets(table(G, perms), mixed), "naive_diff_of_classes", double=double, debug=False)
    # the same members in the same order: the same sums (in double the lists
    # are ascending whatever the order of the call)
    assert a["es"].tobytes() == ref["es"].tobytes()
    if double and G <= 65536:
        assert b["es"].tobytes() == ref["es"].tobytes()
    assert H.es_close(b["es"], ref["es"], double).all()
    for r in (ref, a, b):
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


def test_a_duplicate_costs_nothing_in_double(gpu):
    rs = np.random.RandomState(3)
    clean = [np.sort(rs.choice(20000, size=n, replace=False)) for n in rs.randint(15, 500, 300)]
    plain = es_us(with_sets(table(20000, 304), clean))
    doubled = es_us(with_sets(table(20000, 304), [np.r_[s, s[:1]] for s in clean]))
    # walked in double throughout it took 2.4 times as long
    assert doubled < 1.3 * plain, (doubled, plain)
