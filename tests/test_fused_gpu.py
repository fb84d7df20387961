"""The one-launch build of small and medium clouds against the oracle and the
stage-by-stage build (which the timed entry always runs): sizes at the edges
of its grids, and clouds that drive each of its sorts (bins, radix sort, one
bucket by bitmap) and its tiles."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu
KEYS = ["sorted_unique", "prefix_n", "has_leaf_left", "has_leaf_right", "left_child", "parent",
        "edge_count", "prefix_sum", "oct_nodes"]


def cloud(kind, n, rng):
    pts = np.ones((n, 4), np.float32)
    if kind == "uniform":
        pts[:, :3] = rng.random((n, 3)) * 1023.99
    elif kind == "one bucket":  # 64^3 cells, one value of the top 12 bits: the bitmap
        pts[:, :3] = 512 + rng.random((n, 3)) * 63.99
    elif kind == "bucket and rest":
        pts[:, :3] = rng.random((n, 3)) * 1023.99
        pts[: 3 * n // 4, :3] = 64 + rng.random((3 * n // 4, 3)) * 63.99
    elif kind == "lumps":  # many codes in few bins of a bucket: the radix sort
        pts[:, :3] = rng.integers(0, 16, (n, 3)) * 64 + rng.random((n, 3)) * 6.0
    elif kind == "few cells":
        pts[:, :3] = rng.integers(0, 5, (n, 3)) * 200 + 0.5
    elif kind == "equal":
        pts[:, :3] = 77.25
    else:  # one axis only: long runs of single-child cells
        pts[:, 0] = rng.random(n) * 1023.99
    return pts


def both(pts, n, cap=None):
    """Results of the build and of the stage-by-stage build."""
    from pipeline_gb300 import _lib
    from pipeline_gb300.pipeline import OctreeBuilder

    d = torch.from_numpy(pts).cuda()
    out = []
    for timed in (False, True):
        b = OctreeBuilder(n, cap)
        if timed:
            rc = b.lib.oct_build_octree_timed(
                C.c_void_p(d.data_ptr()), n, 0.0, 1024.0, C.byref(b._out),
                C.c_void_p(b.workspace.data_ptr()), b.workspace.numel(), None, 0,
                C.c_void_p(torch.cuda.current_stream().cuda_stream))
            _lib.check(rc, "oct_build_octree_timed")
        else:
            b.workspace.fill_(0xA5)  # nothing in it may matter
            b.build(d, 0.0, 1024.0)
        out.append(b.result())
    return out


SIZES = [2, 31, 1023, 1025, 4096, 8191, 8193, 20_001, 155_648, 155_649, 400_003]


@pytest.mark.parametrize("kind", ["uniform", "one bucket", "bucket and rest", "lumps", "few cells",
                                  "equal", "one axis"])
def test_matches_oracle_and_stages(kind):
    for n in SIZES:
        pts = cloud(kind, n, np.random.default_rng(n))
        got, staged = both(pts, n, 10 * n + 64)
        want = O.build_all(pts, 0.0, 1024.0)
        assert (got["n_unique"], got["n_oct"], got["status"]) == \
            (want["n_unique"], want["n_oct"], 0), n
        assert staged["n_unique"] == got["n_unique"] and staged["status"] == 0
        if want["n_unique"] < 2:
            continue
        for key in KEYS:
            assert got[key].tobytes() == np.asarray(want[key]).tobytes(), (n, key)
            assert got[key].tobytes() == staged[key].tobytes(), (n, key)


@pytest.mark.parametrize("kind", ["uniform", "bucket and rest"])
def test_largest_share_and_the_first_size_past_it(kind):
    n = torch.cuda.get_device_properties(0).multi_processor_count * 12288
    for m in (n, n + 1):
        got, staged = both(cloud(kind, m, np.random.default_rng(m)), m)
        for key in KEYS:
            assert got[key].tobytes() == staged[key].tobytes(), (m, key)


@pytest.mark.parametrize("n", [3000, 50_000])
def test_status_bits_and_missing_capacity(n):
    pts = cloud("uniform", n, np.random.default_rng(1))
    got, staged = both(pts, n, cap=64)
    assert got["status"] == staged["status"] == 8
    assert (got["n_unique"], got["n_oct"]) == (staged["n_unique"], staged["n_oct"])
    got, staged = both(pts, n, cap=0)
    assert got["prefix_sum"].tobytes() == staged["prefix_sum"].tobytes()
    assert got["n_oct"] == staged["n_oct"]
    pts[n // 2, 1] = np.nan
    pts[n // 3, 0] = -5.0
    got, staged = both(pts, n)
    assert got["status"] == staged["status"] == 4
    for key in KEYS:
        assert got[key].tobytes() == staged[key].tobytes(), key


def test_builds_on_two_streams_at_once():
    from pipeline_gb300.pipeline import OctreeBuilder

    clouds = [cloud("uniform", n, np.random.default_rng(n)) for n in (6000, 300_000)]
    wants = [O.build_all(c, 0.0, 1024.0)["oct_nodes"].tobytes() for c in clouds]
    streams = [torch.cuda.Stream() for _ in clouds]
    builders = [OctreeBuilder(len(c)) for c in clouds]
    inputs = [torch.from_numpy(c).cuda() for c in clouds]
    torch.cuda.synchronize()
    for _ in range(20):
        for b, d, s in zip(builders, inputs, streams):
            b.build(d, 0.0, 1024.0, stream=s)
    torch.cuda.synchronize()
    for b, want in zip(builders, wants):
        assert b.result()["oct_nodes"].tobytes() == want
