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
