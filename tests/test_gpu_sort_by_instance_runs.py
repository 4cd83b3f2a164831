"""The rule by which a batch is sorted instance by instance, seen on the run: a pass of the key
sort is three launches, and all other launches of a batch of these shapes are the same in
number, but for one where some instance has no direct table.  Key widths of 32 and 64 bits on
both sides of the rule, and a batch whose chunks are less than half full."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [8192, 8191, 8193, 16384, 6143, 6145, 12288, 12289, 4097, 24576, 7000, 10241, 8192]
ID_BITS = 4


def _passes(bits):
    digit = 9 if (bits + 8) // 9 < (bits + 7) // 8 else 8
    return -(-bits // digit)


def _batch(sizes, octave):
    rng = np.random.default_rng(octave + 1)
    out = []
    for i, n in enumerate(sizes):
        d = 2 + i % 2
        out.append((rng.uniform(0, 50, (n, d)), (0.25 if d == 2 else 0.4) * 2.0 ** -octave, 3))
    return out


def _launches(ctx, sizes, octave):
    st = ctx.batch_dbscan(_batch(sizes, octave), with_stats=True)[2]
    return st["launches"], st["key_bits"]


@pytest.mark.parametrize("prec", [0, 1])
def test_passes_of_the_run(gpu_ctx, prec):
    gpu_ctx.set_precision(prec)
    seen, rest = set(), set()
    for octave in range(-1, 7):
        launches, bits = _launches(gpu_ctx, SIZES, octave)
        local = bits - ID_BITS
        by_instance = _passes(local) < _passes(bits)
        rest.add(launches - 3 * _passes(local if by_instance else bits))
        seen.add((bits > 32, by_instance))
        # 2,000 points a chunk: the id bits are sorted too
        launches, few = _launches(gpu_ctx, [2000] * len(SIZES), octave)
        rest.add(launches - 3 * _passes(few))
    assert len(rest) <= 2 and max(rest) - min(rest) <= 1
    assert seen == {(False, False), (False, True), (True, False), (True, True)}
