"""The sign of a zero S/N: a sum of one subnormal and a border pixel's scale round to -0.0
or +0.0, which are equal, so that the first motion wins and its zero is the map's. Maps
equal the oracle's bit for bit, signs of zeros included, whatever the tile shape."""
import numpy as np
import pytest

import fainttrail_b200 as ftb


def data(oracle, n=12, w=70, h=37):
    rng = np.random.default_rng(3)
    t = np.linspace(-0.5, 0.5, n)
    grid = 0.5 * np.stack(np.meshgrid(np.arange(-8, 9), np.arange(-8, 9)), -1).reshape(-1, 2)
    frames = np.zeros((n, h, w), np.float32)
    frames[0] = np.where(rng.random((h, w)) < 0.5, np.float32(-1e-45), np.float32(0.0))
    frames[5, 20:] = -1.0
    frames[7, :, 40:] = np.where(rng.random((h, w - 40)) < 0.7, np.float32(-1e-45), np.float32(0.0))
    return frames, t, grid, oracle.shift_table(t, grid)


def bits(a):
    return np.asarray(a, np.float32).view(np.uint32)


@pytest.mark.parametrize("shape", range(9))
def test_plan(oracle, shape):
    frames, t, grid, (dx, dy) = data(oracle)
    for mc in (1, 9):
        want = oracle.stack(frames, dx, dy, mc)
        zero = np.asarray(want[0])[np.asarray(want[0]) == 0]
        assert np.signbit(zero).any() and not np.signbit(zero).all()
        got = ftb.emulate_stack(frames, dx, dy, mc, shape)
        assert np.array_equal(bits(got[0]), bits(want[0])) and np.array_equal(got[1], want[1])


@pytest.mark.gpu
@pytest.mark.parametrize("shape", range(9))
@pytest.mark.parametrize("progress", [False, True])
def test_pass(backend, oracle, shape, progress):
    frames, t, grid, (dx, dy) = data(oracle)
    kw = {"progress": lambda f, s: True} if progress else {}
    try:
        ftb.set_tile_shape(shape)
        for mc in (1, 9):
            want = oracle.stack(frames, dx, dy, mc)
            r = backend.run(ftb.StackPass(frames, t_h=t, velocities=grid, min_count=mc), **kw)
            assert np.array_equal(bits(r.max_snr), bits(want[0])) and np.array_equal(r.best_v, want[1]), mc
    finally:
        ftb.set_tile_shape(0)
