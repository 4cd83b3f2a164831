"""The points belong to the caller once the first expand of an index has run: later expands
must not read them again.  Isolated pairs at eps (1 +/- 1e-7), whose links only the float64
re-test decides, on device points that are overwritten between two expands; sets above the
sizes of the small runs, with direct, row-table and hashed lookups.  Labels against a context
of its own in float64 mode, no tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n,extent", [(2, 270_000, 4e3), (2, 270_000, 1e6), (2, 270_000, 4e7),
                                        (3, 140_000, 200.0), (3, 140_000, 3e3), (3, 140_000, 3e5)])
def test_later_expand_reads_its_own_copy(gpu_ctx, gd, d, n, extent):
    import torch
    rng = np.random.default_rng(d + int(extent))
    a = rng.uniform(0, extent, (n // 2, d))
    v = rng.normal(size=a.shape)
    v /= np.sqrt((v * v).sum(1, keepdims=True))
    b = a + v * (1.0 + 1e-7 * np.where(rng.random((n // 2, 1)) < 0.5, -1.0, 1.0))
    pts = np.concatenate([a, b])[rng.permutation(n)]
    with gd.Context(0, precision=0) as ctx:
        want = [ctx.dbscan(pts, 1.0, mp) for mp in (3, 2)]
    gpu_ctx.set_precision(1)
    t = torch.from_numpy(pts).cuda()
    gpu_ctx.index_build(t, 1.0)
    gpu_ctx.expand(3)
    assert np.array_equal(gpu_ctx.get_result(), want[0])
    t.mul_(0.5)
    torch.cuda.synchronize()
    gpu_ctx.expand(2)
    assert np.array_equal(gpu_ctx.get_result(), want[1])
    st = gpu_ctx.stats()
    if extent < 1e5:
        assert st["precision_used"] == 1 and st["band_retests"] > 0
