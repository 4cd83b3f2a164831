"""Block grid: 64-cell blocks (8x8 in 2D, 4x4x4 in 3D) found directly, through a
table of block rows, or through a hash of rows.  Grids whose sides are just below,
at and above whole blocks, with points in every cell position of a block, against
the oracle; and one context expanding an index several times, where the blocks'
words must start empty again.  Integer labels: no tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(ctx, oracle, pts, eps, mp, prec):
    ctx.set_precision(prec)
    lab, core = ctx.dbscan(pts, eps, mp, with_core=True)
    olab, ocore, _ = oracle.oracle_dbscan(pts, eps, mp)
    assert np.array_equal(core, ocore)
    assert np.array_equal(lab, olab)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("sides", [(1, 1), (7, 9), (8, 8), (9, 17), (1, 40), (33, 3),
                                   (1, 1, 1), (3, 5, 4), (4, 4, 4), (5, 9, 1), (1, 1, 30), (8, 7, 13)])
def test_grid_sides_around_whole_blocks(gpu_ctx, oracle, prec, sides):
    d = len(sides)
    rng = np.random.default_rng(sum(sides) + 100 * d + prec)
    f = 0.5 if d == 2 else 1.0 / np.sqrt(3.0)     # about one cell per unit of f
    n = int(min(4000, 60 + 6 * np.prod(sides)))
    pts = rng.uniform(0, 1, (n, d)) * (np.array(sides) - 0.5) * f
    for mp in (3, 8):
        _check(gpu_ctx, oracle, pts, 1.0, mp, prec)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("d,extent", [(2, 40.0), (2, 3e4), (2, 4e7), (3, 30.0), (3, 600.0), (3, 3e5)])
def test_direct_row_and_hash_lookups(gpu_ctx, oracle, prec, d, extent):
    """Pairs of chains that cross block and row borders, spread over the extent."""
    rng = np.random.default_rng(int(extent) % 1000 + d)
    starts = rng.uniform(0, extent, (60, 1, d))
    steps = rng.normal(0, 0.35, (60, 60, d))
    pts = (starts + np.cumsum(steps, axis=1)).reshape(-1, d)
    pts = pts[rng.permutation(len(pts))]
    for mp in (4, 7):
        _check(gpu_ctx, oracle, pts, 1.0, mp, prec)


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("prec", [0, 1])
def test_expanding_again_after_tuning_changes(gpu_ctx, ds, oracle, prec, graphs):
    """More, then fewer core points on one index, with a tuning change between
    expands (it drops the captured launches but not the index)."""
    inst = ds.blobs2d_100k(seed=9, scale=0.1)
    gpu_ctx.set_precision(prec)
    gpu_ctx.set_graphs(graphs)
    try:
        gpu_ctx.index_build(inst.points, inst.eps)
        for k, mp in enumerate((3, 40, 5, 12, 60)):
            if k in (1, 3):
                gpu_ctx.set_tuning(core_tests=64 + k)
            gpu_ctx.expand(mp)
            assert np.array_equal(gpu_ctx.get_result(),
                                  oracle.oracle_dbscan(inst.points, inst.eps, mp)[0]), mp
    finally:
        gpu_ctx.set_tuning()
        gpu_ctx.set_graphs(True)
