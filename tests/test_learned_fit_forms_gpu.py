"""LearnedCDF.fit where the one-launch Adam steps and the stepwise kernels have
to agree: learning rates that are not positive."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def fit(keys, segments, **kw):
    from pipeline_gb300.learned import LearnedCDF

    return LearnedCDF(max_segments=segments).fit(keys, n_segments=segments, n_buckets=64, **kw)


@pytest.mark.parametrize("lr", [0.0, -0.05, -1.0, float("nan")])
def test_a_rate_that_is_not_positive_moves_nothing(lr):
    """steps * |lr| on both sides of the one-launch form's limit of 16: the model of
    a fit without steps, moments and step count included."""
    rng = np.random.default_rng(3)
    keys = torch.from_numpy(rng.integers(0, 1 << 30, 5000).astype(np.int32)).cuda()
    want, got = fit(keys, 64, steps=0), fit(keys, 64, steps=100, lr=lr)
    assert got.header()["steps"] == want.header()["steps"] == 0
    k = want.header()["n_knots"]
    for name in ("theta", "adam_m", "adam_v"):
        assert got.part(name, np.uint32, k).tobytes() == want.part(name, np.uint32, k).tobytes()


def skewed(kind, n):
    g = torch.Generator(device="cuda").manual_seed(5)
    keys = torch.randint(0, 1 << 30, (n,), generator=g, device="cuda")
    if kind == "one value":
        keys = keys * 0 + 123_456_789
    elif kind == "nine tenths":
        keys[torch.rand(n, generator=g, device="cuda") < 0.9] = 123_456_789
    elif kind == "two values":
        keys = torch.where(keys < 1 << 29, 7, 1 << 29)
    return keys.to(torch.int32)


@pytest.mark.parametrize("kind,segments", [("one value", 1024), ("nine tenths", 1024),
                                           ("nine tenths", 4096), ("two values", 4096),
                                           ("even", 1), ("even", 3)])
def test_long_segments_match_the_fp64_reference(kind, segments):
    """Segments of thousands of keys, summed by chunks of 512 ranks: a short one on
    either side, ends inside a chunk, one segment that is the whole sample. The
    tolerance is that of the one-launch steps (test_learned_fit_gpu.py)."""
    from oracle import learned_ref as LR

    keys = skewed(kind, 40_001)
    m = fit(keys, segments, steps=60, lr=0.05)
    sample = np.sort(keys.cpu().numpy().astype(np.int64))
    x = LR.knots_from_sorted_sample(sample, segments)
    want, _ = LR.adam_fit(sample, x, steps=60, lr=0.05)
    got = m.tables()
    assert np.array_equal(got["x"], x)
    theta = got["theta"].astype(np.float64)
    assert np.linalg.norm(theta - want) <= 1e-4 * np.linalg.norm(want)


def fit_us(keys, segments):
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    best = 1e30
    for _ in range(6):
        torch.cuda.synchronize()
        a.record()
        fit(keys, segments, steps=2)
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b) * 1e3)
    return best


@pytest.mark.parametrize("kind,segments", [("one value", 1024), ("nine tenths", 4096),
                                           ("even", 1)])
def test_no_warp_walks_a_long_segment(kind, segments):
    """One step on a million keys takes no more than three times as long as on even
    keys in short segments (25 to 40 times where one warp walks a segment)."""
    n = 1_000_000
    assert fit_us(skewed(kind, n), segments) < 3 * fit_us(skewed("even", n), 4096)
