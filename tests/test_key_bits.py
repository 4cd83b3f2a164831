"""The float32 position of a coordinate for its cell key is built from the double's
bits: a funnel shift and one flipped exponent bit, zero below 2^-126.  It has to be the
coordinate rounded toward zero over the whole exponent range that the float32 path
admits, and the cells of tiny, zero and negative coordinates the float64 formula's."""
import numpy as np
import pytest


def _from_bits(x):
    b = x.view(np.uint64)
    hw = (b >> np.uint64(32)).astype(np.uint32)
    m = ((b >> np.uint64(29)) & np.uint64(0xffffffff)).astype(np.uint32)   # funnel shift by 3
    m = (m ^ np.uint32(0x40000000)) & np.uint32(0x7fffffff)
    m = np.where((hw & np.uint32(0x7fffffff)) < np.uint32(0x38100000), np.uint32(0), m)
    return ((hw & np.uint32(0x80000000)) | m).astype(np.uint32).view(np.float32)


def test_bits_are_the_truncation():
    rng = np.random.default_rng(11)
    x = rng.uniform(1, 2, 400_000) * 2.0 ** rng.integers(-126, 100, 400_000)
    x = np.concatenate([x, 2.0 ** np.arange(-126.0, 100.0), np.nextafter(2.0 ** np.arange(-125.0, 100.0), 0)])
    x = np.concatenate([x, -x])
    t = x.astype(np.float32)
    over = np.abs(t.astype(np.float64)) > np.abs(x)
    t[over] = np.nextafter(t[over], np.float32(0))
    assert np.array_equal(_from_bits(x), t)
    tiny = np.array([0.0, -0.0, 5e-324, -1e-310, 1e-300, np.nextafter(2.0 ** -126, 0)])
    assert np.all(_from_bits(tiny) == 0)


@pytest.mark.gpu
@pytest.mark.parametrize("d", [2, 3])
@pytest.mark.parametrize("shift", [0.0, -50.0, -99.75])
def test_cells_of_tiny_zero_and_negative_coordinates(gpu_ctx, oracle, d, shift):
    rng = np.random.default_rng(int(-shift) + d)
    pts = rng.uniform(0, 100, (1500, d)) + shift
    special = np.array([0.0, -0.0, 5e-324, 1e-310, -1e-200, 1e-40, 1e-20, -1e-7])
    pts[rng.integers(0, 1500, 300), rng.integers(0, d, 300)] = rng.choice(special, 300)
    pts[:40] = rng.choice(special, (40, d))
    eps = 3.0 if d == 2 else 12.0
    for prec in (0, 1):
        gpu_ctx.set_precision(prec)
        olab, ocore, _ = oracle.oracle_dbscan(pts, eps, 5)
        lab, core = gpu_ctx.dbscan(pts, eps, 5, with_core=True)
        assert np.array_equal(lab, olab) and np.array_equal(core, ocore)
        # the general path: a batch of two
        labels = gpu_ctx.batch_dbscan([(pts, eps, 5), (pts, eps, 5)])
        assert np.array_equal(labels[0], olab) and np.array_equal(labels[1], olab)
