"""Background subtraction with blank growth, and the filter's rescaling, at the edges of
their tiles (128 x 32 pixels, four columns a lane, 16 rows): non-finite pixels at and
near the borders of the image and of the tiles. Searched maps and stages equal the
oracle's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(60, 31), (127, 32), (128, 33), (129, 64), (131, 65), (259, 97)])
def test_blank_growth(device, oracle, w, h):
    rng = np.random.default_rng(w + h)
    n = 6
    mjd = 60000.0 + np.arange(n) / 1440.0
    frames = rng.normal(1000, 10, (n, h, w)).astype(np.float32)
    bad = [(0, 0), (h - 1, w - 1), (0, w - 1), (h - 1, 0), (h // 2, w // 2)]
    bad += [(y, x) for y in (3, 28, 31, 32, 35, 36, 63) for x in (3, 4, 33, 124, 127, 128, 131, 132) if y < h and x < w]
    for i, (y, x) in enumerate(bad):
        frames[i % n, y, x] = (np.nan, np.inf, -np.inf)[i % 3]
    frames[2, 0, 9] = np.float32(3.4e38)
    exp = np.full(n, 30.0)
    got = device.search(frames, mjd, np.zeros(n), fwhm_px=2.0, null_runs=2, vmin_pxh=40.0, vmax_pxh=200.0, min_coverage=0.7)
    sub, _ = oracle.prepare_sub(frames)
    t = (mjd - got["t_ref"]) * 24.0
    filtered = oracle.build_stage(sub, t, 2.0)["filtered"]
    want = oracle.stack(filtered, *oracle.shift_table(t, got["grid"]), oracle.min_count(0.7, n))
    assert np.array_equal(got["max_snr"], want[0], equal_nan=True) and np.array_equal(got["best_v"], want[1])
