"""The run layout of batches around its 1024 instances per round: the grid cells of all block
tables are the sum over the instances, and every instance's labels its own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 1023, 1024, 1025, 2500])
def test_grid_cells_of_all_instances(gpu_ctx, count):
    rng = np.random.default_rng(count)
    insts, want, blocks = [], [], 0
    for i in range(count):
        # two pairs of points at opposite corners of a grid of w blocks (2D: 8 x 8 cells)
        w = rng.integers(1, 9, 2)
        a = (8 * w - 0.5) * 0.5
        insts.append((np.array([[0, 0], [0, 0], a, a, a]), 1.0, int(rng.integers(2, 4))))
        near = a[0] ** 2 + a[1] ** 2 <= 1
        assert not near
        want.append([0, 0, 1, 1, 1] if insts[-1][2] == 2 else [-2, -2, 0, 0, 0])
        blocks += int(w[0] * w[1])
    gpu_ctx.set_precision(0)
    labels, counts, st = gpu_ctx.batch_dbscan(insts, with_stats=True)
    assert st["grid_cells"] == 64 * blocks
    assert all(np.array_equal(a, b) for a, b in zip(labels, want))
