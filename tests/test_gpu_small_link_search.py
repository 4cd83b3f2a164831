"""Small runs: link searches between crowded cells.  Crowds of points a little more than eps
apart, in cells two apart that no bound settles, are never linked, so the search of a pair of
cells runs to its end: by a lane, a warp or the whole grid by the number of point pairs.
Sizes around the borders between the three, a pair that only its last points link, and a
lattice of crowds.  The labels follow from the construction; no tolerance."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _crowds(d, sizes, gap, rng):
    """Crowds along x, `gap` apart (eps 1), and a lone point that sets the grid's origin."""
    lone = np.zeros((1, d))
    lone[0, 1] = 10.0
    pts, who = [lone], [np.full(1, -1)]
    for k, s in enumerate(sizes):
        p = np.full((s, d), 0.15)
        p[:, 0] += k * gap
        pts.append(p + rng.uniform(0, 1e-4, p.shape))
        who.append(np.full(s, k))
    return np.concatenate(pts), np.concatenate(who)


def _expected(who):
    """Labels of groups numbered by their first point; -1: noise."""
    ids, first = np.unique(who, return_index=True)
    rank = {g: r for r, g in enumerate(ids[np.argsort(first)][ids[np.argsort(first)] >= 0])}
    return np.array([rank.get(g, -2) for g in ids])[np.searchsorted(ids, who)]


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("d", [2, 3])
@pytest.mark.parametrize("sizes", [(16, 16), (16, 17), (128, 128), (129, 128), (256, 256),
                                   (256, 257), (257, 5), (362, 362), (363, 362), (1024, 1024),
                                   (1025, 1024), (5, 20_000), (30_000, 30_000), (5000, 7, 5000)])
def test_unlinked_and_last_pair_linked(gpu_ctx, gd, prec, d, sizes):
    rng = np.random.default_rng(sum(sizes) + d)
    pts, who = _crowds(d, sizes, 1.1, rng)
    order = rng.permutation(len(pts))
    gpu_ctx.set_precision(prec)
    lab = gpu_ctx.dbscan(pts[order], 1.0, 4)
    assert gpu_ctx.stats()["launches"] == 3
    assert np.array_equal(lab, _expected(who[order]))
    # one point of the first crowd within eps of one of the second
    pts[1, 0], pts[1 + sizes[0], 0] = 0.2, 1.15
    who[who == 1] = 0
    assert np.array_equal(gpu_ctx.dbscan(pts[order], 1.0, 4), _expected(who[order]))


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("d", [2, 3])
@pytest.mark.parametrize("per,side", [(40, 60), (300, 20), (400, 18)])
def test_lattice_of_crowds(gpu_ctx, prec, d, per, side):
    rng = np.random.default_rng(per + d)
    g = np.stack(np.meshgrid(np.arange(side), np.arange(side), indexing="ij"), -1).reshape(-1, 2)
    site = np.zeros((side * side, d))
    site[:, :2] = 0.15 + 1.1 * g
    who = rng.permutation(np.repeat(np.arange(side * side), per))[: 262144 if d == 2 else 131072]
    pts = site[who] + rng.uniform(0, 1e-4, (len(who), d))
    gpu_ctx.set_precision(prec)
    lab = gpu_ctx.dbscan(pts, 1.0, 4)
    assert gpu_ctx.stats()["launches"] == 3
    assert np.array_equal(lab, _expected(who))


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("d", [2, 3])
def test_without_allocation(built_lib, gd, prec, d):
    import torch
    lib = gd.load_library()
    rng = np.random.default_rng(d)
    pts, who = _crowds(d, (14_000, 14_000, 9), 1.1, rng)
    order = rng.permutation(len(pts))
    t = torch.from_numpy(pts[order]).cuda()
    out = torch.empty(len(pts), dtype=torch.int32, device="cuda")
    k = ctypes.c_int64()
    assert lib.gd_dbscan_noalloc(t.data_ptr(), len(pts), d, 1.0, 4, prec, out.data_ptr(),
                                 ctypes.byref(k), None) == 0
    assert k.value == 3
    assert np.array_equal(out.cpu().numpy(), _expected(who[order]))
