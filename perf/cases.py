"""Performance cases of the octree build: the calls users of this package make,
over the sizes and distributions they make them with.

A case is a dict of plain values; ``prepare`` makes a state from it and a seed
(inputs on the GPU, the builder with its workspace, a fitted model), ``run`` is
one pass through the public entry points, ``work`` the bytes a pass cannot do
without, ``exact`` a 64-bit restatement of the one path with floating-point
results (the model fit; everything else is integers and bytes).

The kinds:

  build      OctreeBuilder: one cloud, every stage, launched on the stream or
             replayed from a CUDA graph
  learned    LearnedOctreeBuilder: the same with the learned bucket sort
  batch      BatchOctreeBuilder: clouds of uneven size in one launch sequence
  frames     BatchOctreeBuilder with a model: scan frames built together
  pipelined  PipelinedBuilder: host frames in, host octrees out
  stages     the per-stage functions in the order a port of the reference's
             driver calls them
  sort       k_SimpleRadixSort alone
  fit        LearnedCDF.fit: knots, Adam steps, bucket tables
"""
from __future__ import annotations

import math

import numpy as np
import torch

from pipeline_gb300 import kernels as K
from pipeline_gb300.batch import BatchOctreeBuilder
from pipeline_gb300.learned import LearnedCDF
from pipeline_gb300.pipeline import LearnedOctreeBuilder, OctreeBuilder, PipelinedBuilder

BOX = 1024.0
TOP = float(np.nextafter(np.float32(BOX), np.float32(0)))
BEAMS, AZIMUTHS = 64, 1920
FRAME = BEAMS * AZIMUTHS  # 122,880 points
TREE = ("prefix_n", "has_leaf_left", "has_leaf_right", "left_child", "parent", "edge_count",
        "prefix_sum")


def listed():
    return [
        # A small object or a leaf region rebuilt on its own: launches and host calls count.
        {"name": "build_4k", "kind": "build", "cloud": "uniform", "n": 4096, "graph": False},
        # One lidar revolution as it arrives, with its own origin and extent.
        {"name": "build_frame", "kind": "build", "cloud": "frame", "n": FRAME, "graph": False},
        # The reference's CPU configuration.
        {"name": "build_uniform_1m", "kind": "build", "cloud": "uniform", "n": 1 << 20,
         "graph": False},
        # The same points captured once and rebuilt every step (the headline workload).
        {"name": "build_uniform_16m", "kind": "build", "cloud": "uniform", "n": 1 << 24,
         "graph": True},
        # An uneven cloud with many points per cell, of a size that fills no tile evenly, near
        # the 10M points of the reference's own benchmark suite.
        {"name": "build_clustered_10m", "kind": "build", "cloud": "clustered", "n": 10_000_003,
         "graph": False},
        # The uneven cloud at full size through the learned bucket sort.
        {"name": "learned_clustered_16m", "kind": "learned", "cloud": "clustered", "n": 1 << 24,
         "graph": False},
        # Hundreds of clouds of 1K to 1M points, half uniform, half mixtures, in one launch.
        {"name": "batch_512", "kind": "batch", "clouds": 512, "lo": 1000, "hi": 1_000_000,
         "graph": True},
        # A recorded drive: frames built together, sorted with a model fit on earlier frames.
        {"name": "frames_224", "kind": "frames", "clouds": 224, "graph": True},
        # A live drive: frames uploaded, built and their octrees downloaded, overlapped.
        {"name": "pipelined_8", "kind": "pipelined", "frames": 8},
        # A caller that keeps the reference's stage-by-stage driver (sizes read on the host).
        {"name": "stages_1m", "kind": "stages", "cloud": "uniform", "n": 1_000_003},
        # The sort alone on full 32-bit keys.
        {"name": "sort_u32_8m", "kind": "sort", "n": 8_388_607, "bits": 32},
        # Fitting the model to a new scene before its first learned build.
        {"name": "fit_4096", "kind": "fit", "n": 262_144, "segments": 4096, "steps": 100},
    ]


def _log_int(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["build", "build", "build", "learned", "batch", "frames", "pipelined",
                       "stages", "sort", "fit"])
    if kind in ("build", "learned"):
        cloud = rng.choice(["uniform", "clustered", "frame"])
        lo = 1000 if kind == "build" else 50_000
        n = FRAME if cloud == "frame" else _log_int(rng, lo, 1 << 24)
        n -= rng.randrange(0, max(n // 16, 1))  # ragged
        return {"kind": kind, "cloud": cloud, "n": n, "graph": rng.random() < 0.5}
    if kind == "batch":
        lo = _log_int(rng, 1000, 20_000)
        hi = _log_int(rng, lo + 1, 1_000_000)
        most = max(8, min(512, int(48e6 / ((lo + hi) / 2))))
        return {"kind": kind, "clouds": _log_int(rng, 8, most), "lo": lo, "hi": hi,
                "graph": rng.random() < 0.5}
    if kind == "frames":
        return {"kind": kind, "clouds": _log_int(rng, 4, 224), "graph": rng.random() < 0.5}
    if kind == "pipelined":
        return {"kind": kind, "frames": rng.randrange(3, 12)}
    if kind == "stages":
        return {"kind": kind, "cloud": rng.choice(["uniform", "clustered"]),
                "n": _log_int(rng, 1000, 10_000_000)}
    if kind == "sort":
        return {"kind": kind, "n": _log_int(rng, 1000, 1 << 24), "bits": rng.choice([30, 32])}
    return {"kind": kind, "n": _log_int(rng, 16_384, 262_144),
            "segments": rng.choice([1024, 2048, 4096]), "steps": rng.randrange(50, 201)}


# ------------------------------------------------------------------ inputs --
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1_000_003 + 17)


def _points(xyz):
    out = torch.ones((xyz.shape[0], 4), dtype=torch.float32, device="cuda")
    out[:, :3] = xyz.clamp(0.0, TOP)
    return out


def _uniform(n, g):
    return torch.rand((n, 3), generator=g, device="cuda") * BOX


def _mixture(n, parts, g):
    """Anisotropic Gaussians: uniform centres, sigma log-uniform in 0.5%..20% of the box."""
    centre = _uniform(parts, g)
    low, high = math.log(0.005), math.log(0.20)
    sigma = BOX * torch.exp(low + (high - low) * torch.rand((parts, 3), generator=g,
                                                           device="cuda"))
    part = torch.randint(0, parts, (n,), generator=g, device="cuda")
    return torch.randn((n, 3), generator=g, device="cuda") * sigma[part] + centre[part]


def _clustered(n, g):
    """64 Gaussians and 5% noise, as heavy in duplicate codes as scanned scenes are."""
    xyz = _mixture(n, 64, g)
    noise = torch.rand((n, 1), generator=g, device="cuda") < 0.05
    return torch.where(noise, _uniform(n, g), xyz)


def _frame(g):
    """64 beams x 1,920 azimuth steps over a ground plane with 40 boxes, 2 cm range noise, in
    scan order. Returns points, and the origin and extent that quantise them."""
    elevation = torch.deg2rad(torch.linspace(-24.8, 2.0, BEAMS, device="cuda"))[:, None]
    azimuth = (torch.arange(AZIMUTHS, device="cuda") * (2 * math.pi / AZIMUTHS))[None, :]
    rays = torch.stack([elevation.cos() * azimuth.cos(), elevation.cos() * azimuth.sin(),
                        elevation.sin().expand(BEAMS, AZIMUTHS)], -1).reshape(-1, 3)
    u = torch.rand((40, 5), generator=g, device="cuda")
    height = 1.8
    centre, half = u[:, :2] * 120 - 60, 0.5 + 3.5 * u[:, 2:4]
    floor = torch.full((40, 1), -height, device="cuda")
    low = torch.cat([centre - half, floor], 1)
    high = torch.cat([centre + half, floor + 1 + 5 * u[:, 4:]], 1)
    t1 = low[:, None, :] / rays[None]
    t2 = high[:, None, :] / rays[None]
    enter = torch.minimum(t1, t2).nan_to_num(-1e30).amax(-1)
    leave = torch.maximum(t1, t2).nan_to_num(1e30).amin(-1)
    hit = (leave >= enter.clamp(min=0)) & (enter > 0)
    t = torch.where(hit, enter, torch.full_like(enter, 120.0)).amin(0)
    down = rays[:, 2] < -1e-6
    t = torch.where(down, torch.minimum(t, -height / rays[:, 2].clamp(max=-1e-6)), t)
    t = t + 0.02 * torch.randn(t.shape, generator=g, device="cuda")
    xyz = rays * t[:, None]
    out = torch.ones((FRAME, 4), dtype=torch.float32, device="cuda")
    out[:, :3] = xyz
    lowest = xyz.min()
    return out, lowest, (xyz.max() - lowest) * (1 + 2.0 ** -16)


def _cloud(case, seed):
    """Points of one cloud, and its origin and extent as host numbers."""
    g, n = _generator(seed), case["n"]
    if case["cloud"] == "frame":
        pts, low, extent = _frame(g)
        return pts[:n].contiguous(), float(low), float(extent)
    return _points(_uniform(n, g) if case["cloud"] == "uniform" else _clustered(n, g)), 0.0, BOX


def _frames(count, g):
    made = [_frame(g) for _ in range(count)]
    return (torch.cat([m[0] for m in made]), torch.stack([m[1] for m in made]),
            torch.stack([m[2] for m in made]))


def _codes(pts, low, extent):
    keys = torch.empty(pts.shape[0], dtype=torch.int32, device="cuda")
    K.k_ComputeMortonCode(pts, keys, pts.shape[0], low, extent)
    return keys


def _sample(keys, count):
    """Every (n / count)-th key, as a program that has just built the scene takes them."""
    at = torch.arange(count, device="cuda") * keys.numel() // count
    return keys[at].contiguous()


def _batch_sizes(case, seed):
    """Sizes log-uniform in [lo, hi]: the same set for every seed, in another order."""
    c, lo, hi = case["clouds"], case["lo"], case["hi"]
    sizes = [int(lo * (hi / lo) ** ((i + 0.5) / c)) for i in range(c)]
    return [sizes[i] for i in np.random.RandomState(seed % (1 << 31)).permutation(c)]


def _batch_points(sizes, g):
    """Even clouds uniform, odd clouds mixtures of 8 Gaussians."""
    parts = [_uniform(n, g) if c % 2 == 0 else _mixture(n, 8, g) for c, n in enumerate(sizes)]
    return _points(torch.cat(parts))


def _outputs(builder, counts):
    """The builder's buffers as they are, whole: zero where no pass writes (past a cloud's own
    counts), as the reference's callers hand them over."""
    out = {name: getattr(builder, name).zero_() for name in TREE + ("codes", "nodes")}
    return dict(out, counts=getattr(builder, counts).zero_())


# ----------------------------------------------------------------- prepare --
def prepare(case, seed):
    return {"build": _prepare_build, "learned": _prepare_build, "batch": _prepare_batch,
            "frames": _prepare_batch, "pipelined": _prepare_pipelined, "stages": _prepare_stages,
            "sort": _prepare_sort, "fit": _prepare_fit}[case["kind"]](case, seed)


def _prepare_build(case, seed):
    pts, low, extent = _cloud(case, seed)
    n = pts.shape[0]
    if case["kind"] == "learned":
        model = LearnedCDF(4096)
        model.fit(_sample(_codes(pts, low, extent), min(n, 262_144)), n_segments=4096, steps=100,
                  n_buckets=4096)
        b = LearnedOctreeBuilder(n, model)
    else:
        b = OctreeBuilder(n)
    out = _outputs(b, "d_counts")
    if case["graph"]:
        b.capture(pts, low, extent)
    return {"kind": "build", "builder": b, "graph": case["graph"], "in": (pts, low, extent),
            "out": out}


def _prepare_batch(case, seed):
    g = _generator(seed)
    model = None
    if case["kind"] == "frames":
        earlier, lows, extents = _frames(16, g)
        sizes = [FRAME] * case["clouds"]
        keys = torch.cat([_codes(earlier[i * FRAME:(i + 1) * FRAME], float(lows[i]),
                                 float(extents[i])) for i in range(16)])
        model = LearnedCDF(1024).fit(_sample(keys, 262_144), n_segments=1024, steps=100,
                                     n_buckets=64)
        pts, lows, extents = _frames(case["clouds"], g)
    else:
        sizes = _batch_sizes(case, seed)
        pts = _batch_points(sizes, g)
        lows = torch.zeros(len(sizes), device="cuda")
        extents = torch.full((len(sizes),), BOX, device="cuda")
    b = BatchOctreeBuilder(sizes, model=model)
    out = _outputs(b, "counts")
    if case["graph"]:
        b.capture(pts, lows, extents)
    return {"kind": "build", "builder": b, "graph": case["graph"], "in": (pts, lows, extents),
            "out": out}


def _prepare_pipelined(case, seed):
    g = _generator(seed)
    frames = []
    for _ in range(case["frames"]):
        pts, low, extent = _frame(g)
        frames.append((pts.cpu().pin_memory(), float(low), float(extent)))
    octrees = [torch.zeros((FRAME, K.OCTNODE_WORDS), dtype=torch.int32).pin_memory()
               for _ in frames]
    return {"kind": "pipelined", "builder": PipelinedBuilder(FRAME), "frames": frames,
            "out": octrees}


def _prepare_stages(case, seed):
    pts, low, extent = _cloud(case, seed)
    n = pts.shape[0]
    word = dict(dtype=torch.int32, device="cuda")
    byte = dict(dtype=torch.uint8, device="cuda")
    s = {"kind": "stages", "pts": pts, "n": n, "low": low, "extent": extent,
         "nodes": K.empty_oct_nodes(n)}
    for name in ("keys", "keys_alt", "codes", "left_child", "parent", "edge_count",
                 "prefix_sum"):
        s[name] = torch.zeros(n, **word)
    for name in ("prefix_n", "has_leaf_left", "has_leaf_right"):
        s[name] = torch.zeros(n, **byte)
    return s


def _prepare_sort(case, seed):
    g, n = _generator(seed), case["n"]
    top = 1 << (case["bits"] - 1)
    keys = torch.randint(-top if case["bits"] == 32 else 0, top if case["bits"] == 32 else 2 * top,
                         (n,), generator=g, device="cuda").to(torch.int32)
    return {"kind": "sort", "from": keys, "keys": torch.empty_like(keys),
            "alt": torch.empty_like(keys), "bits": case["bits"]}


def _fit_sample(case, seed):
    pts = _points(_clustered(4 * case["n"], _generator(seed)))
    return _sample(_codes(pts, 0.0, BOX), case["n"])


def _prepare_fit(case, seed):
    sample = _fit_sample(case, seed)
    model = LearnedCDF(case["segments"])
    model.fit(sample, n_segments=case["segments"], steps=0)
    knots = model.header()["n_knots"]
    theta, heights = (model.blob[model.offsets[p]:model.offsets[p] + 4 * count].view(torch.float32)
                      for p, count in (("theta", knots), ("y", knots + 1)))
    return {"kind": "fit", "model": model, "sample": sample, "segments": case["segments"],
            "steps": case["steps"], "out": {"theta": theta, "heights": heights}}


# --------------------------------------------------------------------- run --
def run(s):
    return {"build": _run_build, "pipelined": _run_pipelined, "stages": _run_stages,
            "sort": _run_sort, "fit": _run_fit}[s["kind"]](s)


def _run_build(s):
    if s["graph"]:
        s["builder"].replay()
    else:
        s["builder"].build(*s["in"])
    return s["out"]


def _run_pipelined(s):
    sizes = s["builder"].run(s["frames"], s["out"])
    s["builder"].synchronize()
    return {"sizes": [list(x) for x in sizes], "octrees": s["out"]}


def _run_stages(s):
    n, low, extent = s["n"], s["low"], s["extent"]
    keys, alt = s["keys"], s["keys_alt"]
    prefix, left, right = s["prefix_n"], s["has_leaf_left"], s["has_leaf_right"]
    child, parent, edges, offsets = s["left_child"], s["parent"], s["edge_count"], s["prefix_sum"]
    K.k_ComputeMortonCode(s["pts"], keys, n, low, extent)
    K.k_SimpleRadixSort(keys, alt, n)
    u = K.k_CountUnique(keys, n)
    codes = s["codes"][:u].copy_(keys[:u])  # kept: the next cloud's keys go to the same buffer
    b = u - 1
    K.k_BuildRadixTree(b, codes, prefix, left, right, child, parent)
    K.k_EdgeCount(prefix, parent, edges, b)
    K.k_PartialSum(edges, 0, b, offsets)
    m = K.octree_node_count(edges, offsets, b)
    nodes = s["nodes"][:m].zero_()
    K.octree_root_init(nodes, codes, prefix, low, extent)
    K.k_MakeOctNodes(nodes, offsets, edges, codes, prefix, parent, low, extent, b)
    K.k_LinkLeafNodes(nodes, offsets, edges, codes, left, right, prefix, parent, child, b)
    return dict({name: s[name] for name in TREE + ("codes", "nodes")}, sizes=[u, b, m])


def _run_sort(s):
    s["keys"].copy_(s["from"])  # the sort is in place: fresh keys for every pass
    K.k_SimpleRadixSort(s["keys"], s["alt"], s["keys"].numel(), key_bits=s["bits"])
    return s["keys"]


def _run_fit(s):
    s["model"].fit(s["sample"], n_segments=s["segments"], steps=s["steps"])
    return s["out"]


# -------------------------------------------------------------------- work --
# Unique codes and OctNodes per point, as the clouds above have them.
PER_POINT = {"uniform": (0.99, 0.47), "clustered": (0.75, 0.34), "frame": (0.23, 0.17)}


def _build_bytes(n, unique, nodes):
    """Points in; per unique code 4 B of codes, 11 B of tree, 8 B of counts and offsets and
    60 B per OctNode out."""
    return n * (16 + 23 * unique + 60 * nodes)


def work(case):
    kind = case["kind"]
    if kind in ("build", "learned", "stages"):
        moved = _build_bytes(case["n"], *PER_POINT[case["cloud"]])
    elif kind == "batch":
        n = sum(_batch_sizes(case, 0))
        moved = _build_bytes(n, 0.95, 0.45)
    elif kind == "frames":
        moved = _build_bytes(case["clouds"] * FRAME, *PER_POINT["frame"])
    elif kind == "pipelined":  # over the host link: points up, OctNodes down
        moved = case["frames"] * FRAME * (16 + 60 * PER_POINT["frame"][1])
    elif kind == "sort":
        moved = 8 * case["n"]
    else:  # the sample in, the parameters and heights out, once
        moved = 4 * case["n"] + 8 * case["segments"]
    return {"bytes": float(moved), "flops": 0.0}


# ------------------------------------------------------------------- exact --
def exact(case, seed):
    """The fit in 64 bits; every other output is a whole number or a byte."""
    if case["kind"] != "fit":
        return None
    v = np.sort(_fit_sample_codes(case, seed))
    count, steps, lr = v.size, case["steps"], 0.05
    at = v[np.arange(case["segments"], dtype=np.int64) * count // case["segments"]]
    x = at[np.concatenate([[True], at[1:] != at[:-1]])]
    k = x.size
    ends = np.concatenate([x[1:], [1 << 30]]).astype(np.float64)
    seg = np.clip(np.searchsorted(x, v, side="right") - 1, 0, k - 1)
    f = np.where(v >= x[0], (v - x[seg]) / (ends[seg] - x[seg]), 0.0)
    target = (np.arange(count) + 0.5) / count
    theta = np.full(k, math.log(math.e - 1.0))
    m, s2 = np.zeros(k), np.zeros(k)

    def heights(theta):
        soft = np.log1p(np.exp(theta))
        return np.concatenate([[0.0], np.cumsum(soft)]) / soft.sum(), soft.sum()

    for step in range(1, steps + 1):
        y, z = heights(theta)
        r = 2.0 * (y[seg] + (y[seg + 1] - y[seg]) * f - target) / count
        g = np.bincount(seg, r * (1.0 - f), k + 1) + np.bincount(seg + 1, r * f, k + 1)
        after = np.cumsum(g[::-1])[::-1]
        grad = (after[1:] - (g * y).sum()) / z / (1.0 + np.exp(-theta))
        m = 0.9 * m + 0.1 * grad
        s2 = 0.999 * s2 + 0.001 * grad * grad
        theta = theta - lr * (m / (1 - 0.9 ** step)) / (np.sqrt(s2 / (1 - 0.999 ** step)) + 1e-8)
    y, _ = heights(theta)
    return {"theta": theta, "heights": y}


def _fit_sample_codes(case, seed):
    """The sample's Morton codes from its points: 10 bits per axis, interleaved."""
    pts = _points(_clustered(4 * case["n"], _generator(seed)))
    pts = pts[torch.arange(case["n"], device="cuda") * pts.shape[0] // case["n"]]
    cell = (pts[:, :3].double() / BOX * 1024.0).floor().long()
    code = torch.zeros(pts.shape[0], dtype=torch.int64, device="cuda")
    for bit in range(10):
        for axis in range(3):
            code |= ((cell[:, axis] >> bit) & 1) << (3 * bit + axis)
    return code.cpu().numpy()
