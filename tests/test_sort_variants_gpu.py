"""The register radix sort alone (sort_variant 3) and the bucket sort with the
radix sorts behind it (0): the same order, ranks and weights at the edges of
every radix class, the same results in a batch whose instances are declined,
taken and tuned to the radix sort alone side by side."""
import ctypes

import numpy as np
import pytest

from cudagsea_gb300 import api, synthetic
from cudagsea_gb300 import _native as N
from tests.test_bucket_sort_gpu import table
from tests.test_parity_gpu import check_sort, run_plan

pytestmark = pytest.mark.gpu

# the last size of every radix class and the first of the next (1,024 threads x
# 4, 8, 12, 16, 20 keys, two-CTA clusters of 16 and 20; doubles 4, 10, clusters of 10)
SIZES = {False: [1, 33, 1000, 4096, 4097, 8192, 8193, 12288, 12289, 16384, 16385, 20480, 20481, 32768, 32769, 40960],
         True: [1, 33, 1000, 4096, 4097, 10240, 10241, 20480]}


def crowded(G, perms, seed=0):
    """Counts: class means a few units apart, hundreds of genes to a value."""
    d = synthetic.make(G, 12, 6, perms, seed=G + seed, n_class_b=6, set_min=5, set_max=min(300, G))
    d.exprs = np.ascontiguousarray(np.random.RandomState(G + seed).poisson(1.5, d.exprs.shape).astype(np.float32))
    return d


@pytest.mark.parametrize("double", [False, True], ids=["f32", "f64"])
@pytest.mark.parametrize("kind", ["plain", "ties", "crowded"])
def test_radix_sort_alone(gpu, kind, double):
    for G in SIZES[double]:
        metric = "naive_diff_of_classes" if kind == "crowded" else "twopass_signal2noise"
        d = table(G, 3, kind)
        asc = bool(G & 1)
        a = run_plan(d, metric, double=double, ascending=asc, tuning=dict(sort_variant=3))
        b = run_plan(d, metric, double=double, ascending=asc)
        check_sort(a["keys"], a["order"], a["ranks"], a["sorted"], ascending=asc)
        for k in ("keys", "order", "ranks", "sorted", "es", "stats"):
            assert a[k].tobytes() == b[k].tobytes(), (G, k)
        with pytest.raises(N.GseaError):  # no bucket sort, nothing left by one
            a["plan"].read_buffer(N.BUF_SORT_LEFT, np.uint8, (3,))
        a["plan"].close()
        b["plan"].close()


@pytest.mark.parametrize("double,G", [(False, 40961), (True, 20481)])
def test_radix_sort_alone_has_its_limits(gpu, double, G):
    d = synthetic.make(G, 8, 3, 4, seed=3, n_class_b=4)
    plan = api.Plan(G, 8, 3, 4, 8, precision=64 if double else 32)
    plan.set_tuning(sort_variant=3)
    plan.set_inputs(d.exprs, d.labels, d.set_offsets, d.set_genes)
    with pytest.raises(N.GseaError):
        plan.execute()
        plan.synchronize()
    plan.close()


class Left:
    """GSEA_BUF_SORT_LEFT of a batch instance."""

    def __init__(self, batch, i):
        self._h = N._p()
        N.check(N.lib().gsea_batch_plan(batch._h, i, self._h))
        self.perms = batch.cfgs[i].num_perms

    def read(self):
        out = np.empty(self.perms, np.uint8)
        N.check(N.lib().gsea_plan_read_buffer(self._h, N.BUF_SORT_LEFT, N.ptr(out), out.nbytes))
        return out


@pytest.mark.parametrize("double", [False, True], ids=["f32", "f64"])
def test_batch_with_declined_instances(gpu, double):
    sizes = [900, 4097, 9000, 13000, 17000, 20480] + ([] if double else [25000, 40000]) + [50000]
    precision = 64 if double else 32
    ds = [crowded(G, 40) for G in sizes] + [synthetic.make(G, 12, 6, 40, seed=G, n_class_b=6, set_max=200)
                                            for G in (1000, 20000)]
    ref = [run_plan(d, "naive_diff_of_classes", double=double) for d in ds]
    b = api.Batch(ds, "naive_diff_of_classes", precision=precision)
    t = N.Tuning()
    N.lib().gsea_tuning_init(ctypes.byref(t))
    t.sort_variant = 3  # one of the crowded instances is tuned to the radix sort alone
    N.check(N.lib().gsea_plan_set_tuning(Left(b, 1)._h, ctypes.byref(t)))
    for _ in range(2):
        b.execute()
        b.synchronize()
        for i, d in enumerate(ds):
            es, st = b.read(i)
            assert es.tobytes() == ref[i]["es"].tobytes(), i
            assert st.tobytes() == ref[i]["stats"].tobytes(), i
    for i in range(len(ds)):
        if i == 1:
            continue
        left = Left(b, i).read()
        assert left.all() if i < len(sizes) else not left.any(), (i, left)
        solo = ref[i]["plan"].read_buffer(N.BUF_SORT_LEFT, np.uint8, (40,))
        assert np.array_equal(left != 0, solo != 0), i
    for r in ref:
        check_sort(r["keys"], r["order"], r["ranks"], r["sorted"])
        r["plan"].close()
    b.close()
