"""Small runs with crowded cells: clumps of very different spread and points at few, Zipf-popular
positions, whose points and cell pairs go from lanes to warps, blocks and the grid.  Direct and
hashed grids, both precisions, the staged call and the call without allocation, against the
oracle.  No tolerance."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _clumps(rng, n, d, box):
    k = max(4, n // 1500)
    centre, spread = rng.uniform(0, box, (k, d)), 10.0 ** rng.uniform(-2.0, 1.0, (k, 1))
    which = rng.integers(0, k, n)
    return centre[which] + spread[which] * rng.normal(size=(n, d))


def _popular(rng, n, d):
    k = max(2, n // 50)
    at = rng.uniform(0, 0.8 * k ** (1.0 / d), (k, d))
    weight = 1.0 / np.arange(1, k + 1)
    return at[rng.choice(k, n, p=weight / weight.sum())]


@pytest.mark.parametrize("d,n", [(2, 700), (2, 12_000), (2, 30_000), (2, 120_000), (3, 700),
                                 (3, 12_000), (3, 30_000), (3, 120_000)])
@pytest.mark.parametrize("kind", ["clumps", "far clumps", "popular"])
def test_crowded_sets(gpu_ctx, gd, oracle, d, n, kind):
    import torch
    rng = np.random.default_rng(n + d)
    if kind == "popular":
        pts, eps = _popular(rng, n, d), 1.0
    else:
        pts, eps = _clumps(rng, n, d, 100.0 if kind == "clumps" or n > 16384 else 3e4), 0.5
    lib = gd.load_library()
    t = torch.from_numpy(pts).cuda()
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    k = ctypes.c_int64()
    for mp in (4, 60, 700):
        lab, core, _ = oracle.oracle_dbscan(pts, eps, mp)
        for prec in (0, 1):
            gpu_ctx.set_precision(prec)
            got, gcore = gpu_ctx.dbscan(pts, eps, mp, with_core=True)
            assert n > 16384 or gpu_ctx.stats()["launches"] == 3
            assert np.array_equal(gcore, core) and np.array_equal(got, lab), (mp, prec)
            if n <= 32768:
                assert lib.gd_dbscan_noalloc(t.data_ptr(), n, d, eps, mp, prec, out.data_ptr(),
                                             ctypes.byref(k), None) == 0
                assert np.array_equal(out.cpu().numpy(), lab), (mp, prec)
