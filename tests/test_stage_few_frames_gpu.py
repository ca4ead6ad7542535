"""Sequences of so few frames that no residual is finite: one frame's scatter map is 0 (the
median of no values), not undefined, so that a mask limit below 0 masks every pixel; two
and more have too few values. Outputs equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 4])
@pytest.mark.parametrize("kw", [{}, {"mask_scatter": -1.0}, {"mask_scatter": 0.0}, {"mask_scatter": -1.0, "weight_scatter": -2.0}])
def test_few_frames(device, oracle, n, kw):
    sub = np.random.default_rng(n).normal(0, 1, (n, 13, 35)).astype(np.float32)
    t = np.linspace(-0.1, 0.1, n)
    got, want = device.stage(sub, t, 1.5, **kw), oracle.build_stage(sub, t, 1.5, **kw)
    for k in ("filtered", "static_sky", "mask", "sigma", "cr"):
        assert np.array_equal(np.asarray(got[k]), np.asarray(want[k]), equal_nan=True), k
