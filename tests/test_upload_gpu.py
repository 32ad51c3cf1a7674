"""An upload that cannot allocate room for its gene sets leaves a plan, and a
batch instance, without inputs: the next execute is refused and launches
nothing on the freed buffers; the next complete upload works again."""
import numpy as np
import pytest

from cudagsea_gb300 import api, synthetic
from cudagsea_gb300 import _native as N

pytestmark = pytest.mark.gpu


def problems():
    small = synthetic.make(600, 12, 8, 40, seed=1, n_class_b=6, set_min=5, set_max=20)
    large = synthetic.make(600, 12, 8, 40, seed=2, n_class_b=6, set_min=100, set_max=200)
    return small, large


def upload(plan, d):
    plan.set_inputs(d.exprs, d.labels, d.set_offsets, d.set_genes)


@pytest.mark.parametrize("precision", [32, 64])
def test_plan_without_sets_is_refused(gpu, monkeypatch, precision):
    small, large = problems()
    plan = api.Plan(600, 12, 8, 40, "naive_diff_of_classes", precision=precision)
    upload(plan, small)
    plan.execute()
    plan.synchronize()
    monkeypatch.setenv("GSEA_FAULT", "alloc")
    with pytest.raises(N.GseaError) as e:
        upload(plan, large)  # more members than there is room for
    assert e.value.status == 8
    monkeypatch.delenv("GSEA_FAULT")
    with pytest.raises(N.GseaError) as e:
        plan.execute()
    assert e.value.status == 1
    upload(plan, large)
    plan.execute()
    es, _ = plan.read()
    ref, _ = api.gsea(large.exprs.astype(plan.dtype), large.labels, large.set_offsets, large.set_genes, 40,
                      "naive_diff_of_classes", precision)
    assert np.array_equal(es, ref)
    plan.close()


def test_batch_instance_without_sets_is_refused(gpu, monkeypatch):
    small, large = problems()
    b = api.Batch([small, small], "naive_diff_of_classes")
    b.execute()
    b.synchronize()
    args = [np.ascontiguousarray(a, t) for a, t in ((large.exprs, np.float32), (large.labels, np.uint8),
                                                    (large.set_offsets, np.int64), (large.set_genes, np.int32))]
    monkeypatch.setenv("GSEA_FAULT", "alloc")
    assert N.lib().gsea_batch_set_inputs(b._h, 1, *map(N.ptr, args)) == 8
    monkeypatch.delenv("GSEA_FAULT")
    with pytest.raises(N.GseaError) as e:
        b.execute()
    assert e.value.status == 1
    N.check(N.lib().gsea_batch_set_inputs(b._h, 1, *map(N.ptr, args)))
    b.execute()
    es, _ = b.read(1)
    ref, _ = api.gsea(large.exprs, large.labels, large.set_offsets, large.set_genes, 40, "naive_diff_of_classes")
    assert np.array_equal(es, ref)
    b.close()


@pytest.mark.parametrize("missing", ["exprs", "labels", "set_genes"])
def test_one_shot_refuses_missing_arrays_before_it_makes_room(gpu, missing):
    """Offsets that ask for more than the device has, and an array missing: the
    missing array is the answer, not the memory."""
    small, _ = problems()
    a = dict(exprs=np.ascontiguousarray(small.exprs, np.float32), labels=np.ascontiguousarray(small.labels, np.uint8),
             set_offsets=np.ascontiguousarray(small.set_offsets, np.int64),
             set_genes=np.ascontiguousarray(small.set_genes, np.int32))
    a["set_offsets"][-1] = 1 << 40
    a[missing] = None
    args = [N.ptr(v) if v is not None else None for v in a.values()]
    es = np.empty((8, 40), np.float32)
    assert N.lib().gsea_run_f32(args[0], 600, 12, args[1], args[2], args[3], 8, 40, 0, 0, N.ptr(es), None, None) == 1
