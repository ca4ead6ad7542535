"""The streamed stacking pass where a plain pass does not lead: the passes of a search, its
null runs and injection copies in one launch, their maxima merged in one buffer; streamed
and resident passes of served requests together; a budget without room for the merged
maxima; a staging wait that runs out. Maps equal the oracle's, and those of the resident
32 x 16 tile, bit for bit."""
import ctypes as C

import numpy as np
import pytest

import fainttrail_b200 as ftb

pytestmark = pytest.mark.gpu


def streamed(w, h, n, dx, dy):
    st = ftb.plan_stats(w, h, n, dx, dy, 0)
    return st["slots"] == st["groups"] * 80


def sequence(seed, n, w, h):
    rng = np.random.default_rng(seed)
    raw = (1000.0 + 30.0 * rng.normal(0, 1, (n, h, w))).astype(np.float32)
    for _ in range(6):
        raw[:, rng.integers(8, h - 8), rng.integers(8, w - 8)] += 2e4
    return raw, 61337.9 + np.arange(n) * 60.0 / 86400.0, np.full(n, 45.0)


def oracle_maps(oracle, raw, mjd, grid):
    t = (mjd - 0.5 * (mjd[0] + mjd[-1])) * 24.0
    filtered = oracle.build_stage(oracle.prepare_sub(raw)[0], t, 2.5)["filtered"]
    dx, dy = oracle.shift_table(t, grid)
    return oracle.stack(filtered, dx, dy, oracle.min_count(0.7, len(mjd))), (dx, dy)


@pytest.mark.parametrize("n,w,h", [(14, 120, 90), (50, 97, 66)])
def test_search_and_batch(device, oracle, n, w, h):
    raw, mjd, exp = sequence(n, n, w, h)
    kw = dict(fwhm_px=2.5, null_runs=3, grid_tol_px=0.125, vmin_pxh=1.0, vmax_pxh=60.0 if n < 20 else 16.0)
    copies = [[(40.0, 40.0, 9.0, -4.0, 900.0)], [(60.5, 30.25, -7.0, 8.0, 1200.0), (20.0, 50.0, 5.0, 5.0, 700.0)]]
    out = {}
    try:
        for shape in (0, 1):
            ftb.set_tile_shape(shape)
            out[shape] = device.search_batch(raw, mjd, exp, copies, **kw)
    finally:
        ftb.set_tile_shape(0)
    want, (dx, dy) = oracle_maps(oracle, raw, mjd, out[0][0]["grid"])
    assert streamed(w, h, n, dx, dy)
    for base, _ in out.values():
        assert np.array_equal(base["max_snr"], want[0]) and np.array_equal(base["best_v"], want[1])
    assert np.array_equal(out[0][0]["null_peaks"], out[1][0]["null_peaks"]) and len(out[0][0]["null_peaks"]) > 0
    for a, b in zip(out[0][1], out[1][1]):
        assert np.array_equal(a["max_snr"], b["max_snr"]) and a["peaks"] == b["peaks"]


def test_served_together(oracle):
    requests = []
    for k, (n, w, h, tol) in enumerate([(14, 120, 90, 0.125), (12, 101, 77, 0.5), (16, 90, 64, 0.125), (13, 140, 80, 0.5)]):
        raw, mjd, exp = sequence(20 + k, n, w, h)
        requests.append((raw, mjd, exp, dict(fwhm_px=2.5, null_runs=2, grid_tol_px=tol, vmin_pxh=1.0, vmax_pxh=60.0)))
    server = ftb.Server(0, max_batch=8, workers=1)
    try:
        tickets = [server.submit(raw, mjd, exp, **kw) for raw, mjd, exp, kw in requests * 3]
        results = [server.poll(t) for t in tickets]
    finally:
        server.close()
    kinds = set()
    for k, (raw, mjd, exp, kw) in enumerate(requests):
        n, h, w = raw.shape
        want, (dx, dy) = oracle_maps(oracle, raw, mjd, results[k]["grid"])
        kinds.add(streamed(w, h, n, dx, dy))
        for r in results[k::len(requests)]:
            assert np.array_equal(r["max_snr"], want[0]) and np.array_equal(r["best_v"], want[1])
    assert kinds == {True, False}


def lattice(oracle, n, w, h):
    rng = np.random.default_rng(n)
    t = np.linspace(-0.5, 0.5, n)
    grid = 0.5 * np.stack(np.meshgrid(np.arange(-16, 17), np.arange(-16, 17)), -1).reshape(-1, 2)
    frames = rng.normal(0, 1, (n, h, w)).astype(np.float32)
    dx, dy = oracle.shift_table(t, grid)
    assert streamed(w, h, n, dx, dy)
    return frames, t, grid, (dx, dy)


def test_no_room_for_merged_maxima(oracle):
    n, w, h = 10, 256, 200
    frames, t, grid, (dx, dy) = lattice(oracle, n, w, h)
    want = oracle.stack(frames, dx, dy, 7)
    held = 4 * n * w * h + 8 * w * h  # frames and maps
    small = ftb.Device(0, held + 4 * w * h)  # not the 8 w h bytes of merged maxima
    try:
        be = ftb.make_backend("b200", small)
        for kw in ({}, {"progress": lambda f, s: True}, {}):  # in steps: by the resident kernel
            r = be.run(ftb.StackPass(frames, t_h=t, velocities=grid, min_count=7), **kw)
            assert np.array_equal(r.max_snr, want[0]) and np.array_equal(r.best_v, want[1])
    finally:
        small.close()


def test_bounded_wait(backend, oracle):
    """Each staging barrier expects 16 bytes that no copy brings: the waits give up after
    about 10 ms, the pass fails with an error, and the context runs the next one."""
    L = ftb.lib()
    L.ft_b200_set_wait_test.argtypes = [C.c_int, C.c_longlong]
    frames, t, grid, (dx, dy) = lattice(oracle, 12, 130, 70)
    p = ftb.StackPass(frames, t_h=t, velocities=grid, min_count=8)
    for kw in ({}, {"progress": lambda f, s: True}):
        try:
            assert L.ft_b200_set_wait_test(16, 20_000_000) == ftb.FT_B200_OK
            with pytest.raises(RuntimeError, match="timed out"):
                backend.run(p, **kw)
        finally:
            assert L.ft_b200_set_wait_test(0, 0) == ftb.FT_B200_OK
        r = backend.run(p)
        want = oracle.stack(frames, dx, dy, 8)
        assert np.array_equal(r.max_snr, want[0]) and np.array_equal(r.best_v, want[1])
