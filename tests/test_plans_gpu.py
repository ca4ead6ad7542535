"""The first search of a size that the autotuner has not seen: the plans of its passes are
made together by the host threads once the shapes are known, not one after another, and
their time is part of the "plans" entry of the timings."""
import os
import time

import numpy as np
import pytest

import fainttrail_b200 as ftb

pytestmark = pytest.mark.gpu


def test_plans_of_an_unseen_size(device, oracle):
    import torch
    n, w, h, passes = 30, 1040, 1016, 8
    mjd = 61337.9 + np.arange(n) * 60.0 / 86400.0
    frames = 1000.0 + 30.0 * torch.randn((n, h, w), generator=torch.Generator("cuda").manual_seed(1), device="cuda")
    kw = dict(vmin_pxh=12.0, vmax_pxh=84.0, grid_tol_px=0.125, fwhm_px=2.5, null_runs=passes - 1)
    ftb.clear_tuned_shapes()
    first = device.search_dev(frames.data_ptr(), w, h, w, n, mjd, np.full(n, 45.0), **kw)
    times = dict(device.timings())
    assert float(len(first["grid"])) * n * w * h > 5e11 and "autotune" in times
    dx, dy = oracle.shift_table((mjd - 0.5 * (mjd[0] + mjd[-1])) * 24.0, first["grid"])
    tuned = ftb.tuned_shapes()[(n, len(first["grid"]), w, h)]
    t0 = time.perf_counter()
    ftb.plan_stats(w, h, n, dx, dy, tuned)
    one = time.perf_counter() - t0
    assert times["plans"] > 0.3 * one
    if (os.cpu_count() or 1) >= passes:
        assert times["plans"] < 0.7 * passes * one
    again = device.search_dev(frames.data_ptr(), w, h, w, n, mjd, np.full(n, 45.0), **kw)
    assert np.array_equal(first["max_snr"], again["max_snr"]) and np.array_equal(first["best_v"], again["best_v"])
    assert first["threshold"] == again["threshold"]
