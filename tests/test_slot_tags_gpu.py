"""Stages 6-8 with slot tags against the oracle where they can go wrong: tiles
with more octree slots than they stage, radix nodes spanning several levels at
tile edges, leaves further off than a link tag holds, clouds of every size of
the tag's distance field, and clouds too large for slot tags (node tags)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu
KEYS = ["sorted_unique", "edge_count", "prefix_sum", "oct_nodes"]


def spread(codes):
    """Points at the centres of Morton cells (unit cells of a 1024 box)."""
    pts = np.ones((len(codes), 4), np.float32)
    for axis in range(3):
        cell = np.zeros(len(codes), np.int64)
        for bit in range(10):
            cell |= ((codes >> (3 * bit + axis)) & 1) << bit
        pts[:, axis] = cell + 0.5
    return pts


def cloud(kind, n, rng):
    if kind == "pairs":  # every other node spans about five levels: over 8,000 slots a tile
        c = rng.integers(0, 1 << 27, n // 2).astype(np.int64) << 3
        codes = np.concatenate([c, c | 1])
    elif kind == "chains":  # pairs, triples and long runs mixed
        c = rng.integers(0, 1 << 20, n // 4).astype(np.int64) << 10
        codes = np.concatenate([c, c | 1, c | 8, c + rng.integers(0, 1 << 10, len(c))])
    elif kind == "comb":  # one leaf far off each range: 0, then a dense run, at every scale
        codes = np.concatenate([np.arange(n - 30), (1 << np.arange(30)).astype(np.int64) - 1])
    else:
        codes = rng.integers(0, 1 << 30, n).astype(np.int64)
    return spread(rng.permutation(codes))


@pytest.mark.parametrize("kind", ["pairs", "chains", "comb", "uniform"])
@pytest.mark.parametrize("n", [64, 4100, 20_000, 140_000])
def test_build_matches_oracle(kind, n):
    from pipeline_gb300.pipeline import OctreeBuilder

    pts = cloud(kind, n, np.random.default_rng(n))
    want = O.build_all(pts, 0.0, 1024.0)
    b = OctreeBuilder(len(pts), 10 * len(pts))
    b.build(torch.from_numpy(pts).cuda(), 0.0, 1024.0)
    got = b.result()
    assert (got["n_oct"], got["status"]) == (want["n_oct"], 0)
    for key in KEYS:
        assert got[key].tobytes() == np.asarray(want[key]).tobytes(), key


def test_batch_matches_oracle():
    from pipeline_gb300.batch import BatchOctreeBuilder

    rng = np.random.default_rng(9)
    clouds = [cloud(k, n, rng) for n in (70, 4099, 30_001) for k in
              ("pairs", "chains", "comb", "uniform")]
    sizes = [len(c) for c in clouds]
    b = BatchOctreeBuilder(sizes, node_caps=[10 * n + 1 for n in sizes])
    b.build(torch.from_numpy(np.concatenate(clouds)).cuda(), torch.zeros(len(sizes)).cuda(),
            torch.full((len(sizes),), 1024.0).cuda())
    for c, pts in enumerate(clouds):
        got, want = b.cloud_result(c), O.build_all(pts, 0.0, 1024.0)
        for key in KEYS:
            assert got[key].tobytes() == np.asarray(want[key]).tobytes(), (c, key)


@pytest.mark.slow
@pytest.mark.parametrize("form", ["single", "batch"])
def test_clouds_past_the_slot_tag_limit_match_oracle(form):
    """The octree of 120,000,001 points over 3,000 cells is that of the cells."""
    from pipeline_gb300.batch import BatchOctreeBuilder
    from pipeline_gb300.pipeline import OctreeBuilder

    few = O.init_random_vec4(3000, seed=4)
    want = O.build_all(few, 0.0, 1024.0)
    n = 120_000_001
    pts = torch.from_numpy(few).cuda()[torch.arange(n, device="cuda") % len(few)]
    if form == "single":
        b = OctreeBuilder(n, 20_000)
        b.build(pts, 0.0, 1024.0)
        got = b.result()
    else:
        b = BatchOctreeBuilder([n], node_caps=[20_000])
        b.build(pts, torch.zeros(1).cuda(), torch.full((1,), 1024.0).cuda())
        got = b.cloud_result(0)
    assert got["status"] == 0
    for key in KEYS:
        assert got[key].tobytes() == np.asarray(want[key]).tobytes(), key
