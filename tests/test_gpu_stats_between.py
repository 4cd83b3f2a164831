"""Statistics asked for between an expand and its result are those of the last finished run:
all its phase times, none of the running one's, and no error left behind."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TIMES = ("ms_index", "ms_core", "ms_label", "ms_total")


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("n", [20_000, 700_000])
def test_stats_between_expand_and_result(gpu_ctx, n, graphs):
    rng = np.random.default_rng(n)
    pts = rng.uniform(0, (n / 30.0) ** 0.5, (n, 2))
    gpu_ctx.set_precision(0)
    gpu_ctx.set_graphs(graphs)
    try:
        # read at once, as the reference for what the phases may take
        gpu_ctx.index_build(pts, 0.3)
        gpu_ctx.expand(5)
        gpu_ctx.get_result()
        first = gpu_ctx.stats()
        gpu_ctx.index_build(pts, 0.3)
        gpu_ctx.expand(5)
        want = gpu_ctx.get_result()
        for mp in (6, 7, 5):
            gpu_ctx.expand(mp)
            st = gpu_ctx.stats()
            assert st["n_clusters"] == (first["n_clusters"] if mp == 6 else last)
            assert all(st[k] > 0 for k in TIMES), st
            assert st["ms_total"] == st["ms_index"] + st["ms_core"] + st["ms_union"] + st["ms_label"]
            lab = gpu_ctx.get_result()
            last = int(lab.max()) + 1
        assert np.array_equal(lab, want)
    finally:
        gpu_ctx.set_graphs(True)
