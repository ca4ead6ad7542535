"""Frame statistics of more clusters than the chip holds at once, with more samples a
frame than a cluster's lists keep: the CTAs of a cluster exchange the sample's bracket
through one another's shared memory while earlier clusters still run, so that they
start at different times. The stage's sigmas equal the oracle's, in every repetition."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,w,h", [(64, 369, 366), (90, 421, 330)])
def test_more_clusters_than_fit(device, oracle, n, w, h):
    rng = np.random.default_rng(n)
    sub = rng.normal(0, 10, (n, h, w)).astype(np.float32)
    sub *= rng.uniform(0.5, 2.0, (n, 1, 1)).astype(np.float32)
    t = np.linspace(-0.2, 0.2, n)
    want = oracle.build_stage(sub, t, 1.5)
    for _ in range(5):
        got = device.stage(sub, t, 1.5)
        assert np.array_equal(got["sigma"], want["sigma"])
        assert np.array_equal(got["filtered"], want["filtered"], equal_nan=True)
