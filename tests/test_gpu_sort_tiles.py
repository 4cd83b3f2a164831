"""The key sort around its tile sizes: a last tile of one pair, whole tiles, and the number
of tiles from which one histogram block takes four (the last of them perhaps empty), with
32-bit and 64-bit keys.  The points are copies of well separated sites in random order, so
the labels follow from the sites' counts and first indices.  No tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BIG = 1024   # tiles


@pytest.mark.parametrize("bits,tile", [(32, 4096), (64, 2048)])
@pytest.mark.parametrize("tiles,extra", [(80, 1), (BIG - 1, 0), (BIG - 1, 1), (BIG, 0), (BIG, 1),
                                         (BIG + 2, 7), (BIG + 3, -1)])
def test_tile_counts(gpu_ctx, bits, tile, tiles, extra):
    n = tiles * tile + extra
    rng = np.random.default_rng(n)
    # 2D: 1200 x 1200 sites; 3D: sites far apart along every axis (keys beyond 32 bits)
    if bits == 32:
        site = rng.integers(0, 1200 * 1200, n)
        pts = np.stack([site // 1200, site % 1200], axis=1) * 4.0
    else:
        site = rng.integers(0, 1 << 20, n)
        pts = np.stack([site >> 14, (site >> 7) & 127, site & 127], axis=1) * np.array([900.0, 901.0, 902.0])
    gpu_ctx.set_precision(1)
    mp = max(2, n // (1200 * 1200 if bits == 32 else 1 << 20))
    lab, core = gpu_ctx.dbscan(pts, 1.0, mp, with_core=True)
    ids, first, inv, cnt = np.unique(site, return_index=True, return_inverse=True, return_counts=True)
    dense = cnt >= mp
    rank = np.full(len(ids), -2, np.int64)
    order = np.argsort(first[dense])
    r = np.empty(len(order), np.int64)
    r[order] = np.arange(len(order))
    rank[dense] = r
    assert np.array_equal(core.astype(bool), dense[inv])
    assert np.array_equal(lab, rank[inv])
