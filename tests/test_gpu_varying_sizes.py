"""One context over runs of very different sizes, small ones before large ones.

The sort's histogram and its scan's status words must not share memory: in one
buffer laid out by the size at hand, a large sort reads the histogram that a
small one left as status words, and a count that looks like a published prefix
sends its scatter out of range.  Labels must be those of a context of its own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,big", [(2, 2_300_000), (3, 1_700_000)])
def test_small_runs_before_large_ones(gd, built_lib, dim, big):
    rng = np.random.default_rng(17 + dim)
    sets = [rng.uniform(0, (n / 40.0) ** (1.0 / dim), (n, dim)) for n in (3_000, 90_000, 400_001, big)]
    eps = 0.25 if dim == 2 else 0.4
    want = []
    for pts in sets:
        with gd.Context(0) as ctx:
            want.append(ctx.dbscan(pts, eps, 8))
    with gd.Context(0) as ctx:
        for _ in range(6):
            for pts, w in zip(sets, want):
                assert np.array_equal(ctx.dbscan(pts, eps, 8), w)
