"""Several expands of one index on the general path, whose blocks' words must start empty again
and whose launches are captured on the second expand: sets above the sizes of the small runs,
with direct, row-table and hashed lookups, more and then fewer core points, a tuning change in
between (it drops the captured launches but not the index).  Labels and core flags against the
oracle, no tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
_want = {}


def _case(d, extent):
    """Clumps and chains that cross block and row borders."""
    n = 270_000 if d == 2 else 140_000
    rng = np.random.default_rng(d + int(extent) % 1000)
    m = n // 100
    start = rng.uniform(0, extent, (m, 1, d))
    step = rng.normal(0, 0.3, (m, 70, d))
    chain = (start + np.cumsum(step, axis=1)).reshape(-1, d)
    clump = (start[:, :, :] + 3.0 + rng.normal(0, 0.25, (m, 30, d))).reshape(-1, d)
    pts = np.concatenate([chain, clump])
    return pts[rng.permutation(len(pts))]


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("d,extent", [(2, 600.0), (2, 1e5), (2, 2e7), (3, 60.0), (3, 600.0), (3, 3e4)])
def test_more_and_fewer_core_points(gpu_ctx, oracle, d, extent, prec, graphs):
    pts = _case(d, extent)
    gpu_ctx.set_precision(prec)
    gpu_ctx.set_graphs(graphs)
    try:
        gpu_ctx.index_build(pts, 1.0)
        for k, mp in enumerate((3, 40, 5, 12, 3, 60)):
            if k in (2, 4):
                gpu_ctx.set_tuning(core_tests=64 + k)
            if (d, extent, mp) not in _want:
                _want[d, extent, mp] = oracle.oracle_dbscan(pts, 1.0, mp)[:2]
            lab, core = _want[d, extent, mp]
            gpu_ctx.expand(mp)
            got, gcore = gpu_ctx.get_result(with_core=True)
            assert np.array_equal(gcore, core) and np.array_equal(got, lab), mp
        assert gpu_ctx.stats()["launches"] > 20
    finally:
        gpu_ctx.set_tuning()
        gpu_ctx.set_graphs(True)
