"""The streamed stacking pass (shape 6) at the edges of its tiles (32 x 16), runs of
frames, groups and work items, against the oracle, bit for bit: its plan walked on
the CPU, and the kernel on the B200, whole and in parts. Integer values make exact
ties, one pixel is NaN."""
import numpy as np
import pytest

import fainttrail_b200 as ftb

# frames, width, height, lattice step in pixels at the sequence's ends, motions at most
CASES = [(1, 32, 16, 0.25, 9), (2, 33, 15, 0.25, 40), (7, 31, 17, 0.2, 300), (33, 64, 33, 0.25, 700),
         (32, 97, 16, 0.15, 500), (120, 65, 31, 0.25, 330), (255, 40, 20, 0.2, 900)]


def table(oracle, n, w, h, step, most):
    rng = np.random.default_rng(n)
    t = np.sort(rng.uniform(0.0, 1.0, n)) if n > 1 else np.zeros(1)
    t = t - 0.5 * (t[0] + t[-1])
    v = step / max(0.5, -t[0]) * np.arange(-40, 41)
    vx, vy = np.meshgrid(v, v)
    keep = np.argsort(np.hypot(vx, vy).ravel(), kind="stable")[:most]
    grid = np.stack([vx.ravel()[np.sort(keep)], vy.ravel()[np.sort(keep)]], 1)
    frames = rng.normal(0, 1, (n, h, w)).astype(np.float32)
    frames[:, 3, :] = np.round(frames[:, 3, :])
    frames[:, 5, 2:9] = -1e-45  # sums and S/N that round to a zero of either sign
    frames[n // 2, 7, 9] = np.nan
    return t, grid, frames, oracle.shift_table(t, grid)


def same(a, b):
    return np.array_equal(np.asarray(a), np.asarray(b), equal_nan=True)


@pytest.mark.parametrize("n,w,h,step,most", CASES)
def test_streamed_plan(oracle, n, w, h, step, most):
    t, grid, frames, (dx, dy) = table(oracle, n, w, h, step, most)
    st = ftb.plan_stats(w, h, n, dx, dy, 6)
    assert st["slots"] == st["groups"] * 80  # a streamed plan: 16 blocks of 5 slots a group
    for mc in (1, max(1, (7 * n) // 10), n):
        ms, bv = ftb.emulate_stack(frames, dx, dy, mc, 6)
        want = oracle.stack(frames, dx, dy, mc)
        assert same(ms, want[0]) and same(bv, want[1]), mc


def test_automatic_choice(oracle):
    """Small images and tall stacks of close motions are streamed; coarse lattices,
    unstructured tables and stacks of more than 255 frames are not."""
    def slots(n, w, h, step):
        dx, dy = table(oracle, n, 40, 20, step, 700)[3]
        st = ftb.plan_stats(w, h, n, dx, dy, 0)
        return st["slots"] == st["groups"] * 80
    assert slots(20, 1024, 1024, 0.25) and slots(49, 4096, 4096, 0.25) and not slots(48, 4096, 4096, 0.25)
    assert not slots(20, 64, 64, 0.8) and not slots(256, 64, 64, 0.25)
    rng = np.random.default_rng(1)
    a = rng.integers(-9, 10, (2, 200, 12)).astype(np.int32)
    st = ftb.plan_stats(64, 64, 12, a[0], a[1], 0)
    assert st["slots"] != st["groups"] * 80


@pytest.mark.gpu
@pytest.mark.parametrize("n,w,h,step,most", CASES)
@pytest.mark.parametrize("progress", [False, True])
def test_streamed_pass(backend, oracle, n, w, h, step, most, progress):
    t, grid, frames, (dx, dy) = table(oracle, n, w, h, step, most)
    kw = {"progress": lambda f, s: True} if progress else {}
    try:
        ftb.set_tile_shape(6)
        for mc in (1, max(1, (7 * n) // 10), n):
            r = backend.run(ftb.StackPass(frames, t_h=t, velocities=grid, min_count=mc), **kw)
            want = oracle.stack(frames, dx, dy, mc)
            assert same(r.max_snr, want[0]) and same(r.best_v, want[1]), mc
    finally:
        ftb.set_tile_shape(0)
