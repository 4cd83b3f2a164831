"""General path: link searches of crowded cells by a warp, with lanes over the points of either
cell.  The crowds of test_gpu_small_link_search.py through a batch, which always takes the
general path: sizes around the borders where a thread hands a pair over and where the lanes
change sides, unlinked and linked by the last points.  The labels follow from the construction;
no tolerance."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from test_gpu_small_link_search import _crowds, _expected  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("d", [2, 3])
def test_crowds_through_a_batch(gpu_ctx, prec, d):
    rng = np.random.default_rng(d)
    insts, want = [], []
    for sizes in ((6, 7), (16, 17), (256, 255), (257, 5), (5, 257), (31, 3000), (3000, 33), (7, 9000),
                  (9000, 7), (700, 700), (2000, 1500), (600, 9, 600)):
        pts, who = _crowds(d, sizes, 1.1, rng)
        order = rng.permutation(len(pts))
        insts.append((pts[order], 1.0, 4))
        want.append(_expected(who[order]))
        # one point of the first crowd within eps of one of the second
        pts, who = pts.copy(), who.copy()
        pts[1, 0], pts[1 + sizes[0], 0] = 0.2, 1.15
        who[who == 1] = 0
        insts.append((pts[order], 1.0, 4))
        want.append(_expected(who[order]))
    gpu_ctx.set_precision(prec)
    for lab, w, inst in zip(gpu_ctx.batch_dbscan(insts), want, insts):
        assert np.array_equal(lab, w), len(inst[0])
