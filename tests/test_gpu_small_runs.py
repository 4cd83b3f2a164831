"""Small runs (one instance in two cooperative kernels) against the general pipeline
(which gd_batch_dbscan always takes) and the oracle: sizes around a warp, a block and
several blocks, direct and hashed grids, the size limits of the small kernels, and
repeated expands.  Integer labels: no tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(rng, n, d, spread):
    k = 1 + n // 300
    c = rng.uniform(0, spread, (k, d))
    return np.concatenate([c[rng.integers(0, k, n - n // 8)] + rng.normal(0, 0.5, (n - n // 8, d)),
                           rng.uniform(0, spread, (n // 8, d))])


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("d", [2, 3])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 127, 128, 129, 511, 512, 513, 1500, 16384])
@pytest.mark.parametrize("spread", [8.0, 3e4])
def test_sizes_and_lookups(gpu_ctx, oracle, prec, d, n, spread):
    rng = np.random.default_rng(n + 7 * d)
    pts = _points(rng, n, d, spread if spread > 100 else spread * (1 + n / 500) ** (1.0 / d))
    for mp in (1, 5, 12):
        gpu_ctx.set_precision(prec)
        lab, core = gpu_ctx.dbscan(pts, 0.3, mp, with_core=True)
        assert gpu_ctx.stats()["launches"] == 3
        olab, ocore, _ = oracle.oracle_dbscan(pts, 0.3, mp)
        assert np.array_equal(core, ocore)
        assert np.array_equal(lab, olab)
        assert np.array_equal(gpu_ctx.batch_dbscan([(pts, 0.3, mp)])[0], lab)


@pytest.mark.parametrize("d,limit", [(2, 262144), (3, 131072)])
@pytest.mark.parametrize("over", [0, 1])
def test_around_the_size_limits(gpu_ctx, d, limit, over):
    n = limit + over
    rng = np.random.default_rng(d)
    pts = _points(rng, n, d, (n / 8.0) ** (1.0 / d))
    gpu_ctx.set_precision(1)
    lab = gpu_ctx.dbscan(pts, 0.3, 6)
    assert (gpu_ctx.stats()["launches"] == 3) == (over == 0)
    assert np.array_equal(gpu_ctx.batch_dbscan([(pts, 0.3, 6)])[0], lab)


def test_heavy_cells_and_duplicates(gpu_ctx, oracle):
    """Few cells of many points, none dense, and a crowd of equal points."""
    rng = np.random.default_rng(5)
    pts = np.concatenate([rng.normal(0, 0.4, (6000, 2)), np.full((3000, 2), 0.25),
                          rng.uniform(-2, 2, (300, 2))])
    for mp in (2000, 4500, 9000):
        for prec in (0, 1):
            gpu_ctx.set_precision(prec)
            lab, core = gpu_ctx.dbscan(pts, 0.5, mp, with_core=True)
            olab, ocore, _ = oracle.oracle_dbscan(pts, 0.5, mp)
            assert np.array_equal(core, ocore)
            assert np.array_equal(lab, olab)


def test_one_directional_pairs(gpu_ctx):
    """A core pair that is a neighbour in one direction only: the merge replay of the
    small expand gives the general pipeline's labels."""
    base = np.array([[1e-20, 0.0], [-0.3, 0.0]])
    for order in ([0, 1], [1, 0]):
        pts = np.concatenate([base[order], base[order] + [0.0, 50.0], [[9.0, 9.0]]])
        for mp in (1, 2):
            gpu_ctx.set_precision(0)
            assert np.array_equal(gpu_ctx.dbscan(pts, 0.3, mp),
                                  gpu_ctx.batch_dbscan([(pts, 0.3, mp)])[0])
