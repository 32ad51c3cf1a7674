"""Host threads whose problems share kernels but not sizes: no launch is
refused because another thread's launch of the same kernel needs less shared
memory, and every result is that of the problem alone."""
import threading

import numpy as np
import pytest

from cudagsea_gb300 import api, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,sizes", [(32, (10300, 12288)), (64, (10300, 12288)), (32, (24600, 32700))])
def test_threads_of_different_sizes(gpu, precision, sizes):
    ds = [synthetic.make(G, 8, 4, 4, seed=G, n_class_b=4, set_min=15, set_max=60) for G in sizes]

    def call(d):
        return api.gsea(d.exprs.astype(np.float64 if precision == 64 else np.float32), d.labels, d.set_offsets,
                        d.set_genes, 4, "twopass_signal2noise", precision)

    ref = [call(d) for d in ds]
    errors = []

    def loop(i):
        try:
            for _ in range(200):
                es, st = call(ds[i])
                assert np.array_equal(es, ref[i][0]) and np.array_equal(st, ref[i][1], equal_nan=True)
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=loop, args=(i % 2,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
