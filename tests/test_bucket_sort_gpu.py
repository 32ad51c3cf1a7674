"""The bucket sort (k_sort_bucket.cu) at the edges of its shapes: order, ranks
and weights equal the oracle's stable sort of the same keys, with ties ranked
by gene, tie buckets, crowded keys (left to the radix sorts), infinities and
NaN, both directions, and several permutations per CTA."""
import numpy as np
import pytest

from cudagsea_gb300 import synthetic
from tests.test_parity_gpu import check_sort, run_plan

pytestmark = pytest.mark.gpu

# the last size of every shape and the first of the next (256 x 8, 512 x 8,
# 512 x 20, 1,024 x 20 keys, then windows), the smallest and the largest
SIZES = [1, 2, 31, 33, 65, 255, 257, 2048, 2049, 4096, 4097, 10240, 10241, 20480, 20481, 30011, 65535, 65536]


def table(G, perms, kind):
    d = synthetic.make(G, 10, 2, perms, seed=G, n_class_b=5, set_min=1, set_max=min(60, G))
    t = G // 3
    if kind == "ties" and G > 3:      # a third constant, some absent, some equal pairs
        d.exprs[:, :t] = 5.0
        d.exprs[:, t:t + t // 4] = 0.0
        d.exprs[:, t + t // 2:t + t // 2 + t // 8] = d.exprs[:, [G - 1]]
    elif kind == "crowded":           # class means a few units in the last place around two values
        d.exprs[:] = np.float32(1.0) + np.float32(2.0 ** -20) * (np.arange(G) % 7).astype(np.float32)
        d.exprs[:, ::2] += d.labels[:, None].astype(np.float32)
        d.exprs += np.float32(2.0 ** -21) * np.random.RandomState(G).randint(0, 8, d.exprs.shape)
    elif kind == "extreme":           # infinities, zeros in ratios, huge and tiny values
        d.exprs[:, : G // 8] = 0.0
        d.exprs[:5, G // 8: G // 4] = 0.0
        d.exprs[:, G // 4: G // 2] *= np.float32(2.0) ** np.linspace(-100, 100, G // 2 - G // 4).astype(np.float32)
    return d


@pytest.mark.parametrize("kind,metric", [("plain", "twopass_signal2noise"), ("ties", "naive_ratio_of_classes"),
                                         ("crowded", "naive_diff_of_classes"),
                                         ("extreme", "naive_ratio_of_classes")])
@pytest.mark.parametrize("double", [False, True], ids=["f32", "f64"])
def test_bucket_sort_is_the_stable_sort(gpu, kind, metric, double):
    for i, G in enumerate(SIZES):
        d = table(G, 3 if G > 30000 else 9 if G > 64 else 700, kind)
        r = run_plan(d, metric, double=double, ascending=bool(i & 1))
        check_sort(r["keys"], r["order"], r["ranks"], r["sorted"], ascending=bool(i & 1))
        r["plan"].close()


@pytest.mark.parametrize("double", [False, True], ids=["f32", "f64"])
def test_bucket_sort_several_permutations_per_cta(gpu, double):
    """More permutations than CTAs: counters, bitmaps and keys loaded ahead
    are those of the permutation at hand, tie buckets and declined ones between."""
    for G, perms in ((1500, 1500), (15000, 400), (21000, 330)):
        d = table(G, perms, "ties")
        r = run_plan(d, "twopass_signal2noise", double=double)
        check_sort(r["keys"], r["order"], r["ranks"], r["sorted"])
        r["plan"].close()
