"""The matched filter at the edges of its tiles (64 columns; 64 - 2 R rows, a multiple of
four) for every compiled radius and the first general one: cosmic rays beside tile
edges, image borders and each other, masked and weighted pixels, clips of either sign.
Filtered frames, masks and cosmic-ray counts equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
S = 2.354820045030949


@pytest.mark.parametrize("radius", range(1, 10))
@pytest.mark.parametrize("w,h", [(47, 40), (64, 63), (65, 61), (131, 125)])
def test_tiles(device, oracle, radius, w, h):
    rng = np.random.default_rng(100 * radius + w)
    n = 7
    sub = rng.normal(0, 1, (n, h, w)).astype(np.float32)
    ys, xs = rng.integers(0, h, 90), rng.integers(0, w, 90)
    edges = [v for v in (0, 1, 2, 47, 48, 51, 52, 55, 56, 59, 60, 61, 62, 63, 64, 65) if v < min(w, h)]
    ys[:40], xs[40:80] = rng.choice(edges, 40), rng.choice(edges, 40)
    sub[rng.integers(0, n, 90), ys, xs] += rng.uniform(8, 60, 90).astype(np.float32)
    sub[2, h // 2, w // 2 - 1:w // 2 + 2] += 30.0  # centres side by side
    sub[3, 5:9, 5:20] = np.nan
    sub[:, 20:23, 30:40] *= 9.0  # scattered: masked or weighted
    t = np.linspace(-0.3, 0.3, n)
    fwhm = (radius - 0.5) * S / 3.0
    for kw in (dict(), dict(clip_sigma=3.0, cr_sigma=2.0, weight_scatter=0.9), dict(clip_sigma=-1.0, cr_sigma=1.0)):
        got, want = device.stage(sub, t, fwhm, **kw), oracle.build_stage(sub, t, fwhm, **kw)
        for k in ("filtered", "mask", "cr"):
            assert np.array_equal(np.asarray(got[k]), np.asarray(want[k]), equal_nan=True), (kw, k)
