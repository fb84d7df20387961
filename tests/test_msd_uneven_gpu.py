"""The MSD form on uneven clouds, whose large top-digit buckets are cut into
parts by value: a bucket just above the cut and one just below the form's
limit, value ranges so dense that a part has more keys than its run's stage or
its threads walk alone, one code many times, parts without keys, whole long
buckets, and a graph replayed over all of them and over a cloud past the
limit."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

N = (1 << 22) + 1237
MEAN = -(-N // 1024)
CUT = 24576  # four means are less
KEYS = ["sorted_unique", "parent", "prefix_sum", "oct_nodes"]


def spread(codes):
    pts = np.ones((len(codes), 4), np.float32)
    for axis in range(3):
        cell = np.zeros(len(codes), np.int64)
        for bit in range(10):
            cell |= ((codes >> (3 * bit + axis)) & 1) << bit
        pts[:, axis] = cell + 0.5
    return pts


def bucket(b, values):
    return (b << 20) + np.asarray(values, np.int64) % (1 << 20)


def cloud(kind):
    rng = np.random.default_rng(len(kind))
    some = lambda n: rng.integers(0, 1 << 20, n)  # noqa: E731
    parts = {
        "edges": [bucket(0, some(CUT + 1)), bucket(1023, some(CUT - 8000))],
        "largest": [bucket(511, some(31 * MEAN))],
        "dense": [bucket(3, np.arange(120_000)), bucket(4, 77 + np.arange(40_000)),
                  bucket(900, (1 << 20) - 1 - np.arange(23_000))],
        "sparse parts": [bucket(7, some(90_000) % 1000), bucket(8, np.full(120_000, 5)),
                         bucket(9, np.where(some(120_000) % 2, 0, (1 << 20) - 1))],
        "long": [bucket(b, some(20_000)) for b in range(40, 140)],
    }[kind]
    seen = np.concatenate(parts)
    rest = rng.integers(0, 1 << 30, N - len(seen))
    codes = np.concatenate([seen, rest])
    return spread(rng.permutation(codes))


def check(got, want, label):
    assert (got["n_unique"], got["n_oct"], got["status"]) == \
        (want["n_unique"], want["n_oct"], 0), label
    for key in KEYS:
        assert got[key].tobytes() == np.asarray(want[key]).tobytes(), (label, key)


@pytest.mark.parametrize("kind", ["edges", "largest", "dense", "sparse parts", "long"])
def test_uneven_cloud_matches_oracle(kind):
    from pipeline_gb300.pipeline import OctreeBuilder

    pts = cloud(kind)
    b = OctreeBuilder(N)
    b.build(torch.from_numpy(pts).cuda(), 0.0, 1024.0)
    got = b.result()
    assert b.sort_form() == 1
    check(got, O.build_all(pts, 0.0, 1024.0), kind)


def test_captured_build_over_cut_whole_and_lsd_clouds():
    from pipeline_gb300.pipeline import OctreeBuilder

    rng = np.random.default_rng(2)
    past = spread(rng.permutation(np.concatenate(
        [bucket(6, rng.integers(0, 1 << 20, 34 * MEAN)),
         rng.integers(0, 1 << 30, N - 34 * MEAN)])))
    even = O.init_random_vec4(N, 0.0, 1024.0, seed=21)
    d_pts = torch.from_numpy(np.ascontiguousarray(even)).cuda()
    b = OctreeBuilder(N)
    b.capture(d_pts, 0.0, 1024.0)
    for pts, form in ((cloud("dense"), 1), (past, 2), (even, 1), (cloud("largest"), 1)):
        d_pts.copy_(torch.from_numpy(np.ascontiguousarray(pts)))
        b.replay()
        got = b.result()
        assert b.sort_form() == form
        check(got, O.build_all(pts, 0.0, 1024.0), form)
