"""Frames of whole numbers, as a camera gives them, with zeros of both signs: the static
sky of many equal values equals the oracle's, signs included, and takes a small multiple of
the time of frames without equal values (once every median that is a zero was looked up
in rank order, eighty times as long for 120 frames)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [20, 40, 64, 100, 120])
def test_whole_numbers(device, oracle, n):
    rng = np.random.default_rng(n)
    w, h = 515, 300
    t = np.linspace(-0.3, 0.3, n)
    base = rng.normal(0, 8, (n, h, w)).astype(np.float32)
    whole = np.round(base)  # -0.0 where a value rounds up to zero
    assert np.signbit(whole[whole == 0]).any()

    def seconds(sub):
        best = []
        for _ in range(4):
            got = device.stage(sub, t, 1.5)
            best.append(dict(device.timings())["static sky + residuals"])
        return got, min(best)

    _, plain = seconds(base)
    got, ties = seconds(whole)
    want = oracle.build_stage(whole, t, 1.5)
    for k in ("static_sky", "filtered", "mask", "sigma"):
        a, b = np.asarray(got[k]), np.asarray(want[k])
        assert np.array_equal(a, b, equal_nan=True), k
        assert np.array_equal(np.signbit(a[a == 0]), np.signbit(b[b == 0])), k
    assert ties < 6 * plain
