"""Shift tables whose motions share no columns, at the edges of the tiles and of the
frame counts at which the automatic shape changes: the plan walked on the CPU and the
kernel on the B200 equal the oracle bit for bit, border coverage included."""
import numpy as np
import pytest

import fainttrail_b200 as ftb

CASES = [(1, 31, 11, 5), (5, 33, 25, 40), (16, 96, 48, 300), (31, 64, 13, 70), (32, 65, 24, 70), (33, 40, 37, 50),
         (64, 48, 20, 30), (255, 33, 17, 9)]


def data(n, w, h, m):
    rng = np.random.default_rng(n * w)
    frames = rng.normal(0, 1, (n, h, w)).astype(np.float32)
    frames[:, 3] = np.round(frames[:, 3])
    frames[n // 2, 5, 9] = np.nan
    t = np.linspace(-1, 1, n) if n > 1 else np.zeros(1)
    coef = rng.uniform(-9, 9, (2, m, 3))
    dx, dy = np.rint(coef[..., :1] + coef[..., 1:2] * t + coef[..., 2:] * t * t).astype(np.int32)
    dx[0], dy[m // 2] = 0, 400
    dx[m // 3] -= 2 * w
    return frames, np.ascontiguousarray(dx), np.ascontiguousarray(dy)


def same(a, b):
    return np.array_equal(np.asarray(a), np.asarray(b), equal_nan=True)


@pytest.mark.parametrize("n,w,h,m", CASES)
def test_plan(oracle, n, w, h, m):
    frames, dx, dy = data(n, w, h, m)
    for mc in (1, max(1, n // 2), n):
        got, want = ftb.emulate_stack(frames, dx, dy, mc, 0), oracle.stack(frames, dx, dy, mc)
        assert same(got[0], want[0]) and same(got[1], want[1]), mc


@pytest.mark.gpu
@pytest.mark.parametrize("n,w,h,m", CASES)
@pytest.mark.parametrize("shape", [0, 1, 5])
def test_pass(backend, oracle, n, w, h, m, shape):
    frames, dx, dy = data(n, w, h, m)
    try:
        ftb.set_tile_shape(shape)
        for mc in (1, max(1, n // 2), n):
            r = backend.run(ftb.StackPass(frames, shifts=(dx, dy), min_count=mc))
            want = oracle.stack(frames, dx, dy, mc)
            assert same(r.max_snr, want[0]) and same(r.best_v, want[1]), mc
    finally:
        ftb.set_tile_shape(0)
