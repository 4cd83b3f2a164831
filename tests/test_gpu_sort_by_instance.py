"""Batches whose instances fill their chunks are sorted instance by instance on the local
key bits where that saves a pass.  Instances of 2D and 3D in turn (the library orders 2D
first), sizes at the edges of tiles (2048, 4096) and chunks (8192), one empty, and eps over
several octaves so that the key width crosses the widths where the rule changes.  Labels
against the oracle, no tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [8192, 8191, 8193, 0, 16384, 6143, 6145, 12288, 12289, 4097, 24576, 7000, 10241, 8192]


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("octave", [0, 1, 2, 3, 4, 5, 6, 8])
def test_sizes_and_key_widths(gpu_ctx, oracle, prec, octave):
    rng = np.random.default_rng(octave)
    insts = []
    for i, n in enumerate(SIZES):
        d = 2 + i % 2
        centres = rng.uniform(0, 50, (40, d))
        pts = centres[rng.integers(0, 40, n)] + rng.normal(0, 0.5, (n, d))
        pts[: n // 5] = rng.uniform(0, 50, (n // 5, d))
        insts.append((pts, (0.25 if d == 2 else 0.4) * 2.0 ** -octave, 4 if octave < 2 else 2))
    gpu_ctx.set_precision(prec)
    labels, counts, st = gpu_ctx.batch_dbscan(insts, with_stats=True)
    assert st["n_points"] == sum(SIZES)
    for (pts, eps, mp), lab, k in zip(insts, labels, counts):
        if len(pts) == 0:
            assert len(lab) == 0
            continue
        want, _, c = oracle.oracle_dbscan(pts, eps, mp)
        assert np.array_equal(lab, want)
        assert k == c["clusters"]


def test_rule_is_reached():
    """Widths of the cases above: some save a pass, some do not."""
    def passes(bits):
        rb = 9 if (bits + 8) // 9 < (bits + 7) // 8 else 8
        return -(-bits // rb)
    saves = set()
    for octave in (0, 1, 2, 3, 4, 5, 6, 8):
        local = 0
        for d, eps in ((2, 0.25), (3, 0.4)):
            side = 55 / (eps * 2.0 ** -octave * (0.5 if d == 2 else 3 ** -0.5))
            blocks = int(np.ceil(side / (8 if d == 2 else 4))) ** d
            local = max(local, (blocks * 64 - 1).bit_length())
        saves.add(passes(local) < passes(local + 4))
    assert saves == {True, False}
