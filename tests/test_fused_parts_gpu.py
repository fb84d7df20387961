"""One-launch builds of clouds that lie in a small part of their box: buckets at and
past the size from which they are cut, dense and sparse parts, parts that a CTA
takes by bitmap, one value in any order, cut buckets beside scattered codes, the
smallest and largest grids; against the oracle, or the stage-by-stage build where
that is as large as the sizes go. And what such a cloud costs beside an even one."""
import ctypes as C

import numpy as np
import pytest
import torch

from conftest import cell_centres
from oracle import oracle as O

pytestmark = pytest.mark.gpu
KEYS = ["sorted_unique", "prefix_n", "has_leaf_left", "has_leaf_right", "left_child", "parent",
        "edge_count", "prefix_sum", "oct_nodes"]
CUT = 32768  # codes of a top-12-bit bucket (2^18 values)


def cloud(kind, n, rng):
    low = 9 << 18
    if kind == "at the cut":
        codes = np.concatenate([low + rng.choice(1 << 18, CUT, replace=False),
                                (11 << 18) + rng.choice(1 << 18, CUT + 1, replace=False),
                                rng.integers(0, 1 << 30, max(n - 2 * CUT - 1, 0))])
    elif kind == "one bucket":
        codes = low + rng.integers(0, 1 << 18, n)
    elif kind == "dense":
        codes = low + 77 + np.arange(n)
    elif kind == "dense part":  # all of the bucket's codes in 2^10 values: bitmap parts
        codes = np.concatenate([low + (5 << 10) + rng.integers(0, 1 << 10, n - n // 8),
                                rng.integers(0, 1 << 30, n // 8)])
    elif kind == "few values":
        codes = np.concatenate([rng.choice(low + rng.integers(0, 1 << 18, 3), n - n // 4),
                                rng.integers(0, 1 << 30, n // 4)])
    elif kind == "pairs":  # nodes that span several levels: more slots than a tile has nodes
        codes = rng.integers(0, 1 << 27, n // 2) << 3
        codes = np.concatenate([codes, codes | 1])
    elif kind == "last bucket":
        codes = (4095 << 18) + (1 << 18) - 1 - rng.integers(0, 1 << 17, n)
    else:  # a few buckets, sparse and dense, and scattered codes
        codes = np.concatenate([(b << 18) + rng.integers(0, 1 << s, n // 6)
                                for b, s in ((0, 18), (1, 9), (2, 18), (4000, 15))]
                               + [rng.integers(0, 1 << 30, n // 3)])
    return cell_centres(rng.permutation(codes))


def build(pts, timed=False):
    from pipeline_gb300 import _lib
    from pipeline_gb300.pipeline import OctreeBuilder

    n, d = len(pts), torch.from_numpy(pts).cuda()
    b = OctreeBuilder(n, 10 * n + 64)
    b.workspace.fill_(0xA5)
    if timed:
        _lib.check(b.lib.oct_build_octree_timed(
            C.c_void_p(d.data_ptr()), n, 0.0, 1024.0, C.byref(b._out),
            C.c_void_p(b.workspace.data_ptr()), b.workspace.numel(), None, 0,
            C.c_void_p(torch.cuda.current_stream().cuda_stream)), "oct_build_octree_timed")
    else:
        b.build(d, 0.0, 1024.0)
    return b.result()


KINDS = ["at the cut", "one bucket", "dense", "dense part", "few values", "pairs", "last bucket",
         "mixed"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [8192, 17_000, 130_001, 400_003])
def test_matches_oracle(kind, n):
    pts = cloud(kind, n, np.random.default_rng(n))
    got, want = build(pts), O.build_all(pts, 0.0, 1024.0)
    assert (got["n_unique"], got["n_oct"], got["status"]) == (want["n_unique"], want["n_oct"], 0)
    for key in KEYS:
        assert got[key].tobytes() == np.asarray(want[key]).tobytes(), key


@pytest.mark.parametrize("kind", KINDS)
def test_largest_grid_matches_the_stages(kind):
    n = torch.cuda.get_device_properties(0).multi_processor_count * 12288 - 5
    pts = cloud(kind, n, np.random.default_rng(7))[:n]
    got, want = build(pts), build(pts, timed=True)
    assert got["status"] == want["status"] == 0
    for key in KEYS:
        assert got[key].tobytes() == want[key].tobytes(), key


def build_us(pts):
    from pipeline_gb300.pipeline import OctreeBuilder

    d = torch.from_numpy(pts).cuda()
    b = OctreeBuilder(len(pts))
    a, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    best = 1e30
    for _ in range(6):
        torch.cuda.synchronize()
        a.record()
        for _ in range(10):
            b.build(d, 0.0, 1024.0)
        e.record()
        e.synchronize()
        best = min(best, a.elapsed_time(e) * 100)
    return best


@pytest.mark.parametrize("kind", ["one bucket", "dense", "few values"])
@pytest.mark.parametrize("n", [120_000, 400_000, 1_000_000])
def test_a_cloud_in_a_corner_costs_no_more_than_twice_an_even_one(kind, n):
    """(One CTA that took a whole bucket: three to seven times.)"""
    rng = np.random.default_rng(1)
    even = cell_centres(rng.integers(0, 1 << 30, n))
    assert build_us(cloud(kind, n, rng)) < 2 * build_us(even)
