"""Small runs from several host threads at once, a context each: their kernels wait for all
blocks of their own launch, and more launches are in flight than fit the GPU side by side.
Every result is that of the run alone; no run falls back (three launches each)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
def test_threads_with_a_context_each(built_lib, gd, ds, prec):
    sets = [ds.blobs2d_100k(seed=3), ds.blobs2d_100k(seed=4, scale=0.02),
            ds.aniso3d_20m(seed=5, scale=0.004)]
    want = []
    with gd.Context(0, precision=prec) as ctx:
        for s in sets:
            want.append(ctx.dbscan(s.points, s.eps, s.minpts))
    wrong = []

    def work(k):
        with gd.Context(0, precision=prec) as ctx:
            for i in range(25):
                s, w = sets[(k + i) % len(sets)], want[(k + i) % len(sets)]
                lab = ctx.dbscan(s.points, s.eps, s.minpts)
                if not np.array_equal(lab, w) or ctx.stats()["launches"] != 3:
                    wrong.append((k, i))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
