"""The one-launch Adam steps of a fit (one cluster, per-segment moments)
against the fp64 reference loop, at its edges: one segment, a CTA's last
thread, several CTAs, segments of one key and of most keys, a one-key sample.

Tolerance on theta: a gradient is a difference of terms up to about 100 times
its size (segment mass against residual), each rounded to 2^-24, so it is off
by about 6e-6 of itself; 60 steps of lr 0.05 carry at most 60 * 0.05 * 6e-6 =
2e-5 into theta of size 0.5: 1e-4 of its norm with a factor of two to spare."""
import numpy as np
import pytest
import torch

from oracle import learned_ref as LR

pytestmark = pytest.mark.gpu
STEPS = 60


def sample(kind, n, rng):
    if kind == "spread":
        keys = rng.integers(0, 1 << 30, n)
    elif kind == "few values":
        keys = rng.integers(0, 40, n) * 7_000_003
    else:  # half the keys in one value, the rest in narrow lumps
        keys = np.where(rng.random(n) < 0.5, 123_456_789,
                        (rng.integers(0, 64, n) << 24) + rng.integers(0, 1 << 12, n))
    return np.sort(keys.astype(np.int64))


@pytest.mark.parametrize("kind", ["spread", "few values", "lumps"])
@pytest.mark.parametrize("n,segments", [(1, 1), (5000, 1), (5000, 511), (20_001, 512),
                                        (20_001, 513), (60_000, 4096)])
def test_fit_matches_fp64_reference(kind, n, segments):
    from pipeline_gb300.learned import LearnedCDF

    keys = sample(kind, n, np.random.default_rng(n + segments))
    d = torch.from_numpy(keys.astype(np.int32)).cuda()
    got = []
    for _ in range(2):
        m = LearnedCDF(max_segments=segments).fit(d, n_segments=segments, steps=STEPS, lr=0.05,
                                                  n_buckets=64)
        got.append(m.tables())
    h = m.header()
    x = LR.knots_from_sorted_sample(keys, segments)
    assert np.array_equal(got[0]["x"], x) and h["steps"] == STEPS
    want, hist = LR.adam_fit(keys, x, steps=STEPS, lr=0.05)
    theta = got[0]["theta"].astype(np.float64)
    assert np.linalg.norm(theta - want) <= 1e-4 * np.linalg.norm(want)
    final, _ = LR.loss_and_grad(want, keys, x)
    assert abs(h["loss"] - final) <= 2e-3 * final + 1e-9
    assert got[0]["theta"].tobytes() == got[1]["theta"].tobytes()  # exact sums: the same again


def test_fit_with_large_steps_takes_the_stepwise_kernels():
    """steps * lr above the fixed point's range: three launches a step."""
    from pipeline_gb300.learned import LearnedCDF

    keys = sample("spread", 20_000, np.random.default_rng(0))
    m = LearnedCDF(max_segments=64).fit(torch.from_numpy(keys.astype(np.int32)).cuda(),
                                        n_segments=64, steps=40, lr=0.5, n_buckets=64)
    x = m.tables()["x"]
    _, hist = LR.adam_fit(keys, x, steps=41, lr=0.5)
    assert m.header()["steps"] == 40
    assert m.header()["loss"] <= 3 * hist[-1] + 1e-9
