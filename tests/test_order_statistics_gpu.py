"""Frame statistics on the B200 where their selection changes its way: sample
counts below and above what a cluster's lists hold, distributions with few distinct
values (which overfill them), missing samples, two samples or none. The stage's
sigmas and filtered frames equal the oracle's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def values(kind, rng, shape):
    v = rng.normal(0, 10, shape)
    if kind == "coarse":  # a handful of distinct values
        v = np.round(v / 12.0)
    elif kind == "constant":
        v = np.full(shape, 3.0)
        v[..., ::97] = rng.normal(0, 1, v[..., ::97].shape)
    elif kind == "ramp":  # values in image order
        v = np.cumsum(np.abs(v), axis=-1) * rng.choice([-1, 1], shape[:-1] + (1,))
    elif kind == "missing":
        v[rng.random(shape) < 0.31] = np.nan
    return v.astype(np.float32)


@pytest.mark.parametrize("kind", ["normal", "coarse", "constant", "ramp", "missing"])
@pytest.mark.parametrize("w,h", [(5, 5), (7, 5), (64, 41), (369, 359), (369, 366), (890, 890), (1203, 700)])
def test_sigma(device, oracle, w, h, kind):
    rng = np.random.default_rng(w * h)
    sub = values(kind, rng, (5, h, w))
    sub[1, : h // 2] = np.nan
    t = np.linspace(-0.2, 0.2, 5)
    got, want = device.stage(sub, t, 1.5), oracle.build_stage(sub, t, 1.5)
    for k in ("sigma", "filtered"):
        assert np.array_equal(np.asarray(got[k]), np.asarray(want[k]), equal_nan=True), k


@pytest.mark.parametrize("n", [5, 8, 9, 40, 63, 65, 97, 113, 128])
def test_windows(device, oracle, n):
    """Leave-out windows from none to the whole sequence on values with long runs of
    equal ones, signed zeros and missing values."""
    rng = np.random.default_rng(n)
    sub = rng.integers(-2, 3, (n, 7, 65)).astype(np.float32)
    sub[:, 1] = rng.normal(0, 1, (n, 65))
    sub[:, 2] = 1.0
    sub[sub == 0] = rng.choice(np.array([0.0, -0.0], np.float32), np.count_nonzero(sub == 0))
    sub[rng.random(sub.shape) < 0.2] = np.nan
    sub[:, 4:, :20] = np.round(rng.normal(0, 40, (n, 3, 20)))
    t = rng.permutation(np.linspace(-0.3, 0.3, n))
    for exclude in (0, 1, 2, n // 8, 15, 16, 31, 32, n // 2, n - 1, n, 10 * n):
        got = device.stage(sub, t, 1.5, static_exclude=exclude)
        want = oracle.build_stage(sub, t, 1.5, static_exclude=exclude)
        for k in ("static_sky", "filtered", "sigma"):
            a, b = np.asarray(got[k]), np.asarray(want[k])
            assert np.array_equal(a, b, equal_nan=True), (exclude, k)
            assert np.array_equal(np.signbit(a[a == 0]), np.signbit(b[b == 0])), (exclude, k)


@pytest.mark.parametrize("n", [5, 8, 17, 40, 64, 65, 100, 128, 131])
@pytest.mark.parametrize("decades", [0.0, 3.0, 30.0])
def test_scatter_scales(device, oracle, n, decades):
    """The temporal scatter's quotients over frames of very different noise, with
    odd and even counts of values: mask and weighted frames equal the oracle's."""
    rng = np.random.default_rng(n)
    sub = rng.normal(0, 1, (n, 24, 66)) * 10.0 ** rng.uniform(-decades, decades, (n, 1, 1))
    sub = sub.astype(np.float32)
    sub[rng.random(sub.shape) < 0.1] = np.nan
    t = np.linspace(-0.3, 0.3, n)
    kw = dict(mask_scatter=1.4, weight_scatter=0.7)
    got, want = device.stage(sub, t, 1.5, **kw), oracle.build_stage(sub, t, 1.5, **kw)
    for k in ("sigma", "mask", "filtered"):
        assert np.array_equal(np.asarray(got[k]), np.asarray(want[k]), equal_nan=True), k
