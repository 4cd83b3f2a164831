"""Performance cases of the clustering library.

Each case is one call (or one short sequence of calls) that a program makes
through the public surface: the Python Context, or the C entry points behind
it.  Point sets are drawn on the GPU from a seed, with the
shapes the library is used on: Gaussian blobs over uniform noise, Zipf-sized
blobs, rotated anisotropic 3D blobs with pairs planted at the eps boundary,
mixtures with eps from the 4th-nearest-neighbour distance, and vehicle tracks
spread over an extent far larger than eps.  Labels are whole numbers, so there
is nothing to compute in higher precision: two correct runs agree exactly.
"""
import ctypes
import importlib
import math

import numpy as np
import torch

PKG = "fast-cuda-gpu-dbscan_gb300"
FP64, FP32_BAND = 0, 1


def listed():
    return [
        # a control loop that clusters one sensor sweep out of reserved memory
        {"name": "noalloc_2d_1k", "op": "noalloc", "layout": "blobs", "dim": 2, "n": 1_200,
         "minpts": 5, "precision": FP32_BAND},
        # the largest sets that entry point takes, 3D, every test in float64
        {"name": "noalloc_3d_30k", "op": "noalloc", "layout": "blobs", "dim": 3, "n": 30_011,
         "minpts": 8, "precision": FP64},
        # the smallest ordinary call: an interactive selection
        {"name": "blobs_2d_1k", "op": "dbscan", "layout": "blobs", "dim": 2, "n": 1_000,
         "minpts": 5, "precision": FP64, "core": False},
        # a typical analysis set, with the core flags
        {"name": "blobs_2d_100k", "op": "dbscan", "layout": "blobs", "dim": 2, "n": 100_000,
         "minpts": 5, "precision": FP64, "core": True},
        # GPS fixes along vehicle routes over a wide area: the grid takes a row table
        {"name": "tracks_2d_1m5", "op": "dbscan", "layout": "tracks", "dim": 2, "n": 1_500_007,
         "extent": 2.0e5, "minpts": 8, "precision": FP64, "core": False},
        # survey lines in 3D over an extent whose rows only fit a hash; ragged size
        {"name": "tracks_3d_300k", "op": "dbscan", "layout": "tracks", "dim": 3, "n": 333_331,
         "extent": 2.0e4, "minpts": 6, "precision": FP64, "core": False},
        # one index, several minPts: the parameter study every user of DBSCAN makes
        {"name": "sweep_2d_1m", "op": "sweep", "layout": "zipf", "dim": 2, "n": 999_983,
         "minpts": "4,8,16,32,64", "precision": FP32_BAND},
        # the 10M-point 2D set, every test in float64
        {"name": "zipf_2d_10m", "op": "dbscan", "layout": "zipf", "dim": 2, "n": 10_000_000,
         "minpts": 8, "precision": FP64, "core": False},
        # the 20M-point 3D set with pairs at eps (1 +/- 1e-7), float32 filter and band
        {"name": "aniso_3d_20m", "op": "dbscan", "layout": "aniso", "dim": 3, "n": 20_000_000,
         "minpts": 10, "precision": FP32_BAND, "core": False},
        # host arrays in, host labels out, one call
        {"name": "host_3d_2m", "op": "host", "layout": "aniso", "dim": 3, "n": 2_000_001,
         "minpts": 10, "precision": FP32_BAND},
        # a modest batch from host arrays, float64, 2D and 3D mixed
        {"name": "batch_host_64", "op": "batch_host", "count": 64, "lo": 256, "hi": 20_000,
         "precision": FP64},
        # thousands of independent instances in one run, device memory
        {"name": "batch_4096", "op": "batch", "count": 4096, "lo": 256, "hi": 200_000,
         "precision": FP32_BAND},
    ]


def _log_int(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    op = rng.choice(["noalloc", "dbscan", "dbscan", "dbscan", "sweep", "host", "batch_host",
                     "batch"])
    case = {"op": op, "precision": rng.choice([FP64, FP32_BAND])}
    if op in ("batch", "batch_host"):
        if op == "batch":
            case.update(count=_log_int(rng, 128, 3000), lo=256, hi=_log_int(rng, 20_000, 200_000))
        else:
            case.update(count=_log_int(rng, 4, 64), lo=256, hi=_log_int(rng, 2_000, 50_000))
        return case
    dim = rng.choice([2, 3])
    top = {"noalloc": 32_768, "dbscan": 20_000_000, "sweep": 3_000_000, "host": 5_000_000}[op]
    low = {"noalloc": 100, "dbscan": 500, "sweep": 20_000, "host": 5_000}[op]
    layout = rng.choice(["blobs", "zipf", "tracks"] if dim == 2 else ["blobs", "aniso", "tracks"])
    n = _log_int(rng, low, top)
    case.update(layout=layout, dim=dim, n=n)
    if layout == "tracks":
        case["n"] = min(n, 4_000_000)
        case["extent"] = math.exp(rng.uniform(math.log(2e3), math.log(2e5 if dim == 2 else 2e4)))
    if op == "sweep":
        case["minpts"] = ",".join(str(m) for m in sorted(
            rng.sample([3, 4, 6, 8, 12, 16, 24, 32, 48, 64], 4)))
    else:
        case["minpts"] = rng.choice([3, 4, 5, 8, 10, 16, 24, 32])
    if op == "dbscan":
        case["core"] = rng.random() < 0.4
    return case


# ---------------------------------------------------------------- point sets
class _Gen:
    """Uniform and normal draws on the GPU from one seed."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed))

    def rand(self, *shape):
        return torch.rand(*shape, generator=self.g, device="cuda", dtype=torch.float64)

    def randn(self, *shape):
        return torch.randn(*shape, generator=self.g, device="cuda", dtype=torch.float64)

    def pick(self, weights, n):
        edges = torch.cumsum(weights / weights.sum(), 0)
        return torch.searchsorted(edges, self.rand(n)).clamp_(max=weights.numel() - 1)


def _blobs(g, n, dim):
    """20 isotropic blobs, 10% uniform noise, densities of the 100,000-point set."""
    side = 100.0 * (n / 100_000) ** 0.5 if dim == 2 else 30.0 * (n / 100_000) ** (1.0 / 3.0)
    centres = side * g.rand(20, dim)
    sigma = side * (0.005 + 0.015 * g.rand(20, 1)) * (1.0 if dim == 2 else 2.0)
    which = (20 * g.rand(n)).long().clamp_(max=19)
    pts = centres[which] + sigma[which] * g.randn(n, dim)
    noise = g.rand(n) < 0.1
    return torch.where(noise[:, None], side * g.rand(n, dim), pts), 0.5


def _zipf(g, n):
    """500 Zipf-sized 2D blobs, 5% uniform noise, densities of the 10M-point set."""
    side = 1000.0 * math.sqrt(n / 1e7)
    centres = side * g.rand(500, 2)
    sigma = 0.5 * torch.pow(10.0, g.rand(500, 1))
    if n < 1_000_000:  # keep the blobs apart in a small domain
        sigma = sigma * math.sqrt(n / 1e6)
    which = g.pick(torch.arange(1, 501, device="cuda", dtype=torch.float64) ** -1.1, n)
    pts = centres[which] + sigma[which] * g.randn(n, 2)
    noise = g.rand(n) < 0.05
    return torch.where(noise[:, None], side * g.rand(n, 2), pts), 0.3


def _aniso(g, n):
    """64 rotated 3D blobs, 10% noise, 1% of the points in pairs at eps (1 +/- 1e-7)."""
    eps = 0.05
    shrink = (n / 2e7) ** (1.0 / 3.0)
    side = 10.0 * shrink
    centres = side * g.rand(64, 3)
    axes = torch.linalg.qr(g.randn(64, 3, 3).cpu())[0].cuda()
    axes = axes * ((0.02 + 0.48 * g.rand(64, 1, 3)) * shrink)
    which = (64 * g.rand(n)).long().clamp_(max=63)
    z = g.randn(n, 3)
    pts = centres[which] + sum(z[:, k:k + 1] * axes[which, :, k] for k in range(3))
    noise = g.rand(n) < 0.1
    pts = torch.where(noise[:, None], side * g.rand(n, 3), pts)
    pairs = n // 200
    if pairs:
        d = g.randn(pairs, 3)
        d = d / d.square().sum(1, keepdim=True).sqrt()
        factor = 1.0 + 1e-7 * torch.where(g.rand(pairs, 1) < 0.5, -1.0, 1.0).double()
        pts[pairs:2 * pairs] = pts[:pairs] + eps * factor * d
        pts = pts[torch.randperm(n, generator=g.g, device="cuda")]
    return pts.contiguous(), eps


def _tracks(g, n, dim, extent):
    """Random-walk tracks of 200 fixes, steps about eps / 2, jitter, an extent of
    ``extent`` eps per axis."""
    per = 200
    m = (n + per - 1) // per
    eps = 1.0
    start = extent * eps * g.rand(m, 1, dim)
    step = 0.15 * g.randn(m, 1, dim) + 0.2 * g.randn(m, per, dim)
    stay = (g.rand(m, per, 1) > 0.2).double()  # a fifth of the fixes at standstill
    pts = start + torch.cumsum(step * stay, 1) + 0.05 * g.randn(m, per, dim)
    pts = pts.reshape(-1, dim)[:n]
    return pts[torch.randperm(n, generator=g.g, device="cuda")].contiguous(), eps


def _points(case, seed):
    g = _Gen(seed)
    n, dim = case["n"], case["dim"]
    if case["layout"] == "blobs":
        return _blobs(g, n, dim)
    if case["layout"] == "zipf":
        return _zipf(g, n)
    if case["layout"] == "aniso":
        return _aniso(g, n)
    return _tracks(g, n, dim, case["extent"])


def _shapes(case, seed):
    """Sizes (log-uniform), dimensions and minPts of a batch's instances.  Sizes
    and dimensions are the case's own, so that every seed has the same outputs'
    shapes."""
    count = case["count"]
    own = np.random.Generator(np.random.PCG64(count * 1_000_003 + case["hi"]))
    n = np.exp(own.uniform(math.log(case["lo"]), math.log(case["hi"]), count)).astype(int)
    dim = np.where(own.uniform(size=count) < 0.5, 2, 3)
    rng = np.random.Generator(np.random.PCG64(seed))
    return n.tolist(), dim.tolist(), rng.integers(4, 33, count).tolist(), rng


def _mixtures(case, seed):
    """Instances of 1-32 blobs with 5-20% noise, eps the median 4th-neighbour
    distance of a sample.  One flat device tensor, and (n, dim, eps, minpts)."""
    n, dim, minpts, rng = _shapes(case, seed)
    g = _Gen(seed)
    flat = torch.empty(sum(a * b for a, b in zip(n, dim)), dtype=torch.float64, device="cuda")
    med, at = [], 0
    for a, b in zip(n, dim):
        k = int(rng.integers(1, 33))
        centres = 100.0 * g.rand(k, b)
        sigma = 0.5 * torch.pow(10.0, g.rand(k, 1))
        which = g.pick(-torch.log(g.rand(k)) + 1e-9, a)
        pts = centres[which] + sigma[which] * g.randn(a, b)
        noise = g.rand(a) < float(rng.uniform(0.05, 0.20))
        pts = torch.where(noise[:, None], 100.0 * g.rand(a, b), pts)
        flat[at:at + a * b] = pts.reshape(-1)
        at += a * b
        # the points come in random order: the first 32 are a sample
        d2 = sum((pts[:32, None, c] - pts[None, :, c]).square() for c in range(b))
        med.append(torch.topk(d2, 5, dim=1, largest=False).values[:, 4].sqrt().median())
    eps = torch.stack(med).tolist()
    return flat, list(zip(n, dim, eps, minpts))


def _split(flat, inst):
    out, at = [], 0
    for n, dim, eps, minpts in inst:
        out.append((flat[at:at + n * dim].reshape(n, dim), eps, minpts))
        at += n * dim
    return out


# ------------------------------------------------------------------- the calls
def prepare(case, seed):
    gd = importlib.import_module(PKG)
    st = {"case": case, "gd": gd}
    op = case["op"]
    if op in ("batch", "batch_host"):
        flat, inst = _mixtures(case, seed)
        if op == "batch":
            api = importlib.import_module(PKG + ".api")
            desc = (api.GdInstance * len(inst))()
            for d, (n, dim, eps, minpts) in zip(desc, inst):
                d.n, d.dim, d.minpts, d.eps = n, dim, minpts, eps
            ctx = ctypes.c_void_p()
            lib = gd.load_library()
            assert lib.gd_ctx_create(0, ctypes.byref(ctx)) == 0
            assert lib.gd_ctx_set_precision(ctx, case["precision"]) == 0
            total = sum(i[0] for i in inst)
            st.update(lib=lib, ctx=_Handle(lib, ctx), desc=desc, points=flat, count=len(inst),
                      labels=torch.empty(total, dtype=torch.int32, device="cuda"),
                      clusters=np.zeros(len(inst), dtype=np.int64))
        else:
            st["inst"] = [(p.cpu().numpy(), eps, mp) for p, eps, mp in _split(flat, inst)]
            st["ctx"] = gd.Context(0, precision=case["precision"])
    else:
        st["points"], st["eps"] = _points(case, seed)
        if op == "noalloc":
            st["lib"] = gd.load_library()
            st["labels"] = torch.empty(case["n"], dtype=torch.int32, device="cuda")
        else:
            st["ctx"] = gd.Context(0, precision=case["precision"])
        if op == "sweep":
            st["sweep"] = [int(m) for m in case["minpts"].split(",")]
        if op == "host":
            st["points"] = st["points"].cpu().pin_memory()
    torch.cuda.synchronize()
    return st


class _Handle:
    """Owns a C context."""

    def __init__(self, lib, ctx):
        self.lib, self.ctx = lib, ctx

    def __del__(self):
        self.lib.gd_ctx_destroy(self.ctx)


def run(st):
    case = st["case"]
    op = case["op"]
    if op == "dbscan":
        return st["ctx"].dbscan(st["points"], st["eps"], case["minpts"], with_core=case["core"])
    if op == "sweep":
        ctx, pts = st["ctx"], st["points"]
        ctx.index_build(pts, st["eps"])
        out = []
        for minpts in st["sweep"]:
            ctx.expand(minpts)
            out.append(ctx.get_result(out=torch.empty(pts.shape[0], dtype=torch.int32,
                                                      device=pts.device)))
        return out
    if op == "host":
        return st["ctx"].dbscan_fused(st["points"], st["eps"], case["minpts"])[0]
    if op == "noalloc":
        clusters = ctypes.c_int64()
        status = st["lib"].gd_dbscan_noalloc(
            st["points"].data_ptr(), case["n"], case["dim"], st["eps"], case["minpts"],
            case["precision"], st["labels"].data_ptr(), ctypes.byref(clusters), None)
        if status != 0:
            raise RuntimeError(st["lib"].gd_last_error().decode())
        return [st["labels"], clusters.value]
    if op == "batch":
        status = st["lib"].gd_batch_dbscan(
            st["ctx"].ctx, st["count"], st["desc"], st["points"].data_ptr(), 1,
            st["labels"].data_ptr(), st["clusters"].ctypes.data, None)
        if status != 0:
            raise RuntimeError(st["lib"].gd_last_error().decode())
        return [st["labels"], st["clusters"]]
    return st["ctx"].batch_dbscan(st["inst"])


def exact(case, seed):
    """Labels are whole numbers: equal or wrong."""
    return None


def work(case):
    """Coordinates read once, labels (and core flags) written once; one distance per point."""
    if case["op"] in ("batch", "batch_host"):
        # expected size of a log-uniform instance, half of them 2D and half 3D
        lo, hi = case["lo"], case["hi"]
        n = case["count"] * (hi - lo) / math.log(hi / lo)
        return {"bytes": int(n * (8 * 2.5 + 4)), "flops": int(n * 7)}
    n, d = case["n"], case["dim"]
    times = case["minpts"].count(",") + 1 if case["op"] == "sweep" else 1
    out = 4 * times + (1 if case.get("core") else 0)
    return {"bytes": n * (8 * d + out), "flops": n * (3 * d - 1) * times}
