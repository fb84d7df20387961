"""The bucket sort of batched builds against the oracle: buckets larger than a
CTA sorts, alone in a unit, over several units and at a cloud's ends, parts of
them that are counted, one code many times, clouds of one point and of none."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

KEYS = ["sorted_unique", "parent", "prefix_sum", "oct_nodes"]


def spread(codes):
    pts = np.ones((len(codes), 4), np.float32)
    for axis in range(3):
        cell = np.zeros(len(codes), np.int64)
        for bit in range(10):
            cell |= ((codes >> (3 * bit + axis)) & 1) << bit
        pts[:, axis] = cell + 0.5
    return pts


def cloud(kind, rng):
    some = lambda n: rng.integers(0, 1 << 20, n)  # noqa: E731
    codes = {
        "even": rng.integers(0, 1 << 30, 40_000),
        "small": rng.integers(0, 1 << 30, 40),
        "point": np.array([12345]),
        "none": np.zeros(0, np.int64),
        "one bucket": (77 << 20) + some(45_000),
        "first and last": np.concatenate([some(20_000), (1023 << 20) + some(8193),
                                          rng.integers(0, 1 << 30, 10_000)]),
        "counted part": np.concatenate([(5 << 20) + (3 << 12) + some(30_000) % 4096,
                                        (5 << 20) + some(9_000)]),
        "one code": np.concatenate([np.full(25_000, 999), rng.integers(0, 1 << 30, 7_000)]),
        "dense": (8 << 20) + np.arange(49_000),
    }[kind]
    return spread(rng.permutation(codes))


@pytest.mark.parametrize("graph", [False, True])
def test_batch_matches_oracle(graph):
    from pipeline_gb300.batch import BatchOctreeBuilder

    rng = np.random.default_rng(11)
    kinds = ["even", "one bucket", "none", "first and last", "point", "counted part", "small",
             "one code", "dense", "even"]
    clouds = [cloud(k, rng) for k in kinds]
    sizes = [len(c) for c in clouds]
    b = BatchOctreeBuilder(sizes, [10 * n + 10 for n in sizes])
    pts = torch.from_numpy(np.concatenate(clouds)).cuda()
    mins = torch.zeros(len(clouds), device="cuda")
    ranges = torch.full((len(clouds),), 1024.0, device="cuda")
    if graph:
        b.capture(pts, mins, ranges)
        b.replay()
    else:
        b.build(pts, mins, ranges)
    for i, pts_i in enumerate(clouds):
        if len(pts_i) == 0:
            continue
        got, want = b.cloud_result(i), O.build_all(pts_i, 0.0, 1024.0)
        assert got["n_unique"] == want["n_unique"], kinds[i]
        if want["n_unique"] > 1:
            for key in KEYS:
                assert got[key].tobytes() == np.asarray(want[key]).tobytes(), (kinds[i], key)
