"""Stacks of more frames than a byte counts (256 and up, which only tiles of four rows
hold): on tiles that the image's edges cut, where every frame covers a part of the tile,
each pixel's covering frames are still counted exactly. Maps equal the oracle's bit for
bit, for motions with and without shared columns, whole and in progress steps."""
import numpy as np
import pytest

import fainttrail_b200 as ftb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,w,h", [(255, 40, 21), (256, 64, 21), (257, 33, 6), (300, 70, 23), (340, 31, 9)])
@pytest.mark.parametrize("kind", ["lattice", "table"])
def test_many_frames(backend, oracle, n, w, h, kind):
    rng = np.random.default_rng(n)
    frames = rng.normal(0, 1, (n, h, w)).astype(np.float32)
    if kind == "lattice":
        t = np.linspace(-0.5, 0.5, n)
        grid = 1.3 * np.stack(np.meshgrid(np.arange(-3, 4), np.arange(-3, 4)), -1).reshape(-1, 2)
        dx, dy = oracle.shift_table(t, grid)
    else:
        dx, dy = (rng.integers(-5, 6, (40, n)).astype(np.int32) for _ in range(2))
    for mc in (1, (7 * n) // 10, n - 3, n):
        want = oracle.stack(frames, dx, dy, mc)
        for kw in ({}, {"progress": lambda f, s: True}):
            r = backend.run(ftb.StackPass(frames, shifts=(dx, dy), min_count=mc), **kw)
            assert np.array_equal(r.max_snr, want[0]) and np.array_equal(r.best_v, want[1]), (mc, kw)
