"""Passes in a row through one context, whose descriptors come to lie at one address with
other frames, sizes and pitches each time, from buffers that are given back in between:
every pass reads its own frames, streamed and resident kernels alike, alone and in
progress steps. Maps equal the oracle's bit for bit."""
import numpy as np
import pytest

import fainttrail_b200 as ftb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [1, 5, 6, 7])
def test_alternating_passes(device, oracle, shape):
    import torch
    rng = np.random.default_rng(shape)
    sizes = [(9, 64, 48), (14, 97, 33), (9, 48, 64), (21, 40, 90)]
    grid = 0.5 * np.stack(np.meshgrid(np.arange(-12, 13), np.arange(-12, 13)), -1).reshape(-1, 2)
    passes = []
    for n, w, h in sizes:
        t = np.linspace(-0.5, 0.5, n)
        dx, dy = oracle.shift_table(t, grid)
        frames = rng.normal(0, 1, (n, h, w)).astype(np.float32)
        mc = max(1, (7 * n) // 10)
        passes.append((n, w, h, t, dx, dy, mc, frames, oracle.stack(frames, dx, dy, mc)))
    backend = ftb.make_backend("b200", device)
    try:
        ftb.set_tile_shape(shape)
        for k in range(12):
            n, w, h, t, dx, dy, mc, frames, want = passes[(k * 3) % 4]
            pitch = (w + 3) // 4 * 4 + 4 * (k % 3)
            d = torch.zeros((n, h, pitch), device="cuda")
            d[:, :, :w] = torch.from_numpy(frames).cuda()
            ms = torch.empty((h, w), device="cuda")
            bv = torch.empty((h, w), dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            device.stack_dev(d.data_ptr(), w, h, pitch, n, dx, dy, mc, ms.data_ptr(), bv.data_ptr())
            assert np.array_equal(ms.cpu().numpy(), want[0]) and np.array_equal(bv.cpu().numpy(), want[1]), k
            if k % 4 == 3:
                r = backend.run(ftb.StackPass(frames, t_h=t, velocities=grid, min_count=mc),
                                progress=lambda f, s: True)
                assert np.array_equal(r.max_snr, want[0]) and np.array_equal(r.best_v, want[1]), k
            del d, ms, bv
            torch.cuda.empty_cache()
    finally:
        ftb.set_tile_shape(0)
