"""Clouds of neighbours far apart: a radix node spans several octree levels, so a
tile of the prefix sum covers two and more times the slots that it stages at once.
Results against the oracle (single, batched) and against the stages (one launch),
and what such trees cost beside even clouds of as many points."""
import ctypes as C
import statistics

import numpy as np
import pytest
import torch

from conftest import cell_centres
from oracle import oracle as O

pytestmark = pytest.mark.gpu
KEYS = ["sorted_unique", "edge_count", "prefix_sum", "oct_nodes"]


def pairs(n, low, seed=3):
    """Codes c and c | 1 with c over the top bits: the larger `low`, the fewer places."""
    c = np.random.default_rng(seed).integers(0, 1 << (30 - low), n // 2) << low
    return np.concatenate([c, c | 1])


@pytest.mark.parametrize("n,low", [(9000, 3), (60_000, 3), (200_001, 6), (2_000_003, 3)])
def test_batched_and_single_builds_match_oracle(n, low):
    from pipeline_gb300.batch import BatchOctreeBuilder
    from pipeline_gb300.pipeline import OctreeBuilder

    pts = cell_centres(pairs(n, low))
    want = O.build_all(pts, 0.0, 1024.0)
    b = OctreeBuilder(len(pts), 8 * len(pts))
    b.build(torch.from_numpy(pts).cuda(), 0.0, 1024.0)
    both = [b.result()]
    assert (both[0]["n_oct"], both[0]["status"]) == (want["n_oct"], 0)
    sizes = [len(pts), 700]
    bb = BatchOctreeBuilder(sizes, node_caps=[8 * m for m in sizes])
    bb.build(torch.from_numpy(np.concatenate([pts, pts[:700]])).cuda(), torch.zeros(2).cuda(),
             torch.full((2,), 1024.0).cuda())
    both.append(bb.cloud_result(0))
    for got in both:
        for key in KEYS:
            assert got[key].tobytes() == np.asarray(want[key]).tobytes(), key


def steps_us(codes):
    from pipeline_gb300 import _lib
    from pipeline_gb300.pipeline import OctreeBuilder

    pts, n = torch.from_numpy(cell_centres(codes)).cuda(), len(codes)
    b = OctreeBuilder(n, 4 * n)
    lib, stream = b.lib, torch.cuda.current_stream()
    count = lib.oct_build_step_count()
    names = [lib.oct_build_step_name(k).decode() for k in range(count)]
    rows = []
    for _ in range(8):
        events = [torch.cuda.Event(enable_timing=True) for _ in range(count)]
        for e in events:
            e.record(stream)
        torch.cuda.synchronize()
        handles = (C.c_void_p * count)(*[e.cuda_event for e in events])
        _lib.check(lib.oct_build_octree_timed(
            pts.data_ptr(), n, 0.0, 1024.0, C.byref(b._out), b.workspace.data_ptr(),
            b.workspace.numel(), handles, count, stream.cuda_stream), "oct_build_octree_timed")
        torch.cuda.synchronize()
        rows.append([events[k - 1].elapsed_time(events[k]) * 1e3 for k in range(1, count)])
    assert b.result()["status"] == 0
    return {name: statistics.median(r[k] for r in rows) for k, name in enumerate(names[1:])}


def test_deep_trees_cost_by_their_nodes():
    """6M points in pairs have 3.4 times the octree nodes of as many even ones: prefix
    sum and finalize take no more than three and a half times as long (3.9 times
    when a tile left the slots beyond its stage to a search in finalize)."""
    n = 6_000_000
    even = steps_us(np.random.default_rng(1).integers(0, 1 << 30, n))
    deep = steps_us(pairs(n, 3))
    for step in ("prefix sum", "octree finalize"):
        assert deep[step] < 3.5 * even[step], (deep, even)
