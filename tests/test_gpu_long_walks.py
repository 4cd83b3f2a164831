"""Core walks and border searches that look at most of their stencil: uniform sets of 2 to 30
points per cell with minPts about the mean number of neighbours, so that half the points are
core and almost all others border points; and clumps of very different spread, whose crowded
cells go to the warp kernels.  Above the small runs' sizes, both precisions, two budgets of
tests per thread.  Labels and core flags against the oracle, no tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n", [(2, 270_000), (3, 140_000)])
@pytest.mark.parametrize("per", [2, 4, 9, 30])
def test_uniform_sets_at_the_mean(gpu_ctx, oracle, d, n, per):
    f = 0.5 if d == 2 else 3 ** -0.5
    rng = np.random.default_rng(per + d)
    pts = rng.uniform(0, f * (n / per) ** (1.0 / d), (n, d))
    mean = per / f ** d * (np.pi if d == 2 else 4.0 / 3.0 * np.pi)
    for mp in (int(mean), int(1.2 * mean)):
        lab, core, _ = oracle.oracle_dbscan(pts, 1.0, mp)
        for prec in (0, 1):
            gpu_ctx.set_precision(prec)
            for tests in (256, 30):
                gpu_ctx.set_tuning(core_tests=tests, border_tests=tests)
                try:
                    got, gcore = gpu_ctx.dbscan(pts, 1.0, mp, with_core=True)
                finally:
                    gpu_ctx.set_tuning()
                assert gpu_ctx.stats()["launches"] > 20
                assert np.array_equal(gcore, core) and np.array_equal(got, lab), (mp, prec, tests)


@pytest.mark.parametrize("d,n", [(2, 300_000), (3, 150_000)])
@pytest.mark.parametrize("mp", [5, 50, 300])
def test_clumps_of_different_spread(gpu_ctx, oracle, d, n, mp):
    rng = np.random.default_rng(mp + d)
    k = 60
    centre, spread = rng.uniform(0, 100, (k, d)), 10.0 ** rng.uniform(-1.3, 0.7, (k, 1))
    which = rng.integers(0, k, n)
    pts = centre[which] + spread[which] * rng.normal(size=(n, d))
    lab, core, _ = oracle.oracle_dbscan(pts, 0.5, mp)
    for prec in (0, 1):
        gpu_ctx.set_precision(prec)
        for tests in (256, 30):
            gpu_ctx.set_tuning(core_tests=tests, border_tests=tests)
            try:
                got, gcore = gpu_ctx.dbscan(pts, 0.5, mp, with_core=True)
            finally:
                gpu_ctx.set_tuning()
            assert np.array_equal(gcore, core) and np.array_equal(got, lab), (prec, tests)
