"""The bucket sort takes a table whatever order its genes are in: sorted by
scale, by abundance or by effect, no permutation is left to the radix sorts
(GSEA_BUF_SORT_LEFT), and the order is the oracle's."""
import numpy as np
import pytest

from cudagsea_gb300 import synthetic
from cudagsea_gb300 import _native as N
from tests.test_parity_gpu import check_sort, run_plan

pytestmark = pytest.mark.gpu


def table(G, kind, perms):
    d = synthetic.make(G, 20, 2, perms, seed=G, n_class_b=10, set_min=1, set_max=60)
    rs = np.random.RandomState(G + 1)
    noise = rs.standard_normal((20, G))
    if kind == "scale":
        x = 8 + noise * np.sort(rs.lognormal(0, 2, G))
    elif kind == "abundance":
        x = np.sort(rs.lognormal(2, 2, G)) * (1 + 0.3 * noise)
    else:  # the observed permutation's keys ascend with the gene
        x = 8 + 0.05 * noise + np.where(d.labels[:, None] == 1, np.linspace(-3, 3, G)[None, :], 0.0)
    d.exprs = np.ascontiguousarray(x.astype(np.float32))
    return d


@pytest.mark.parametrize("kind", ["scale", "abundance", "effect"])
@pytest.mark.parametrize("double", [False, True], ids=["f32", "f64"])
def test_gene_order_does_not_matter(gpu, kind, double):
    # every shape of the bucket sort: one row of threads, partial last rows,
    # whole rows, windows
    for G in (200, 900, 1024, 2048, 3001, 4096, 10240, 12001, 20000, 20480, 30011, 60000, 65535):
        d = table(G, kind, 6)
        r = run_plan(d, "naive_diff_of_classes", double=double)
        left = r["plan"].read_buffer(N.BUF_SORT_LEFT, np.uint8, (6,))
        assert not left.any(), (G, left)
        check_sort(r["keys"], r["order"], r["ranks"], r["sorted"])
        r["plan"].close()
