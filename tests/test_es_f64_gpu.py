"""Double-precision enrichment (k_es.cuh, find_extremum): the score is taken at
the hit that the walk in fp32 finds, or, where fp32 cannot tell the candidates
apart, by the procedure in double.  Against the oracle's running sum, at the
sizes where the bitmap's words per lane change and for sets whose candidates
tie, lie at the ends of the list or do not exist."""
import numpy as np
import pytest

import oracle
from cudagsea_gb300 import synthetic
from tests import helpers as H
from tests.test_parity_gpu import check_sort, run_plan

pytestmark = pytest.mark.gpu


def sets_of(G, rng):
    """Ends, everything, everything but one, nothing, and random sizes."""
    sets = [np.arange(G), np.arange(G - 1), np.arange(1, G), np.array([0]), np.array([G - 1]), np.array([], int),
            np.array([0, G - 1])]
    sets += [rng.choice(G, size=min(G, n), replace=False) for n in (2, 3, 15, 31, 33, 100, 500, G // 2 + 1)]
    return [s.astype(np.int32) for s in sets]


def case(G, kind, perms=24):
    d = synthetic.make(G, 12, 1, perms, seed=G, n_class_b=6, set_min=1, set_max=1)
    rng = np.random.RandomState(G)
    sets = sets_of(G, rng)
    if kind == "ties":        # few distinct expression rows: equal weights, equal steps
        d.exprs[:] = d.exprs[:, rng.randint(0, min(G, 5), G)]
    elif kind == "mirror":    # gene g + G/2 is gene g mirrored: both signs, the same magnitudes
        h = G // 2
        d.exprs[:, h:2 * h] = 16.0 - d.exprs[:, :h]
        sets += [np.r_[s, s + h].astype(np.int32) for s in (rng.choice(max(h, 1), size=min(max(h, 1), n), replace=False)
                                                            for n in (1, 20, 200)) if h]
    elif kind == "zero":      # constant genes: weights of zero, sets without any weight
        d.exprs[:, : (G + 1) // 2] = 8.0
        sets += [np.arange((G + 1) // 2, dtype=np.int32)]
    d.set_offsets = np.r_[0, np.cumsum([s.size for s in sets])].astype(np.int64)
    d.set_genes = np.concatenate(sets).astype(np.int32)
    return d


def extrema_tie(sk, order, members):
    """The running sum's largest and smallest values are equal in magnitude: either sign is the score."""
    hit = np.isin(order, members)
    w = np.where(hit, np.abs(sk), 0.0)
    rs = np.cumsum(w / w.sum() - ~hit / max(1, (~hit).sum()))
    return abs(max(rs.max(), 0.0) + min(rs.min(), 0.0)) < 1e-11


def scores_match(d, metric):
    r = run_plan(d, metric, double=True)
    sk, order = check_sort(r["keys"], r["order"], r["ranks"], r["sorted"])
    es_o = oracle.es(sk, order, d.set_offsets, d.set_genes)
    r["plan"].close()
    ok = H.es_close(r["es"], es_o, True)
    for k, p in np.argwhere(~ok):
        members = d.set_genes[d.set_offsets[k]:d.set_offsets[k + 1]]
        ok[k, p] = H.es_close(r["es"][k, p], -es_o[k, p], True) and extrema_tie(sk[p], order[p], members)
    bad = np.argwhere(~ok)
    assert bad.size == 0, [(tuple(b), r["es"][tuple(b)], es_o[tuple(b)]) for b in bad[:5]]


# one gene, a lane's first words, and each class of words per lane with its successor
@pytest.mark.parametrize("G", [1, 2, 31, 32, 33, 1023, 1025, 2049, 8193, 12289, 20481, 32769, 40961])
def test_scores_by_size(gpu, G):
    scores_match(case(G, "plain"), "naive_diff_of_classes")


@pytest.mark.parametrize("kind", ["ties", "mirror", "zero"])
@pytest.mark.parametrize("G", [64, 1500, 20000])
def test_scores_that_fp32_cannot_decide(gpu, G, kind):
    scores_match(case(G, kind), "naive_diff_of_classes")


@pytest.mark.parametrize("scale", [2.0 ** -120, 2.0 ** 122])
def test_weights_outside_fp32(gpu, scale):
    """Weights whose sum is tiny or overflows in fp32."""
    d = case(1500, "plain")
    d.exprs *= np.float32(scale)
    scores_match(d, "naive_diff_of_classes")
