"""The motions and track points of a result in one call each equal the calls for one
motion and one point; the counts come without a buffer."""
import ctypes as C

import numpy as np
import pytest

import fainttrail_b200 as ftb

pytestmark = pytest.mark.gpu


def test_arrays_equal_single_calls(device):
    from conftest import golden
    g = golden("search_small.npz")
    L, raw = device.L, np.ascontiguousarray(g["raw"], np.float32)
    seen = {}
    free = L.ft_b200_result_free

    class Spy:
        def __getattr__(self, name):
            return getattr(L, name)

        def ft_b200_result_free(self, r):
            v, p = (C.c_double * 2)(), (C.c_double * 5)()
            m = L.ft_b200_result_velocities(r, None, 0)
            nf = L.ft_b200_result_track_points(r, None, 0)
            nc = L.ft_b200_result_candidates(r, None, None, 0)
            one, at = [], lambda a, k: C.cast(C.byref(a, 8 * k), C.POINTER(C.c_double))
            for j in range(m):
                assert L.ft_b200_result_velocity(r, j, at(v, 0), at(v, 1)) == ftb.FT_B200_OK
                one.append((v[0], v[1]))
            points = []
            for c in range(nc):
                for f in range(nf):
                    assert L.ft_b200_result_track_point(r, c, f, *[at(p, k) for k in range(5)]) == ftb.FT_B200_OK
                    points.append(list(p))
            assert L.ft_b200_result_velocity(r, m, at(v, 0), at(v, 1)) != ftb.FT_B200_OK
            seen.update(grid=np.array(one), points=np.array(points).reshape(nc, nf, 5))
            free(r)

    device.L = Spy()
    try:
        r = device.search(raw, g["mjd"], g["exptime"], fwhm_px=2.5, null_runs=2, threshold_snr=4.0)
    finally:
        device.L = L
    assert len(r["candidates"]) > 0 and np.array_equal(r["grid"], seen["grid"]) and np.array_equal(r["track_points"], seen["points"])
