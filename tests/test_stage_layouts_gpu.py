"""Device frames in layouts that the stage reads and writes directly: row pitches with and
without 16-byte rows, bases off a 16-byte boundary, outputs over the inputs, frames
without noise (which are not rescaled). Outputs equal the oracle's, padding untouched."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,pitch,offset", [(64, 33, 64, 0), (64, 33, 64, 1), (67, 17, 68, 0), (67, 17, 67, 3), (41, 50, 96, 2)])
@pytest.mark.parametrize("over", [False, True])
@pytest.mark.parametrize("n", [7, 130])
def test_layouts(device, oracle, w, h, pitch, offset, over, n):
    import torch
    rng = np.random.default_rng(w + pitch)
    sub = rng.normal(0, 1, (n, h, w)).astype(np.float32)
    sub[2] = 0.0
    sub[:, 4, 5:9] = np.nan
    t = np.linspace(-0.3, 0.3, n)
    src = torch.full((n * h * pitch + 8,), 7.0, device="cuda")
    frames = src[offset:offset + n * h * pitch].view(n, h, pitch)
    frames[:, :, :w] = torch.from_numpy(sub).cuda()
    dst = src if over else torch.full_like(src, 7.0)
    out = dst[offset:offset + n * h * pitch].view(n, h, pitch)
    torch.cuda.synchronize()
    got = device.stage_dev(frames.data_ptr(), w, h, pitch, n, t, 2.0, out.data_ptr())
    want = oracle.build_stage(sub, t, 2.0)
    assert np.array_equal(out[:, :, :w].cpu().numpy(), want["filtered"], equal_nan=True)
    assert np.array_equal(got["sigma"], want["sigma"]) and np.array_equal(got["cr"], want["cr"])
    assert torch.all(out[:, :, w:] == 7.0) and torch.all(dst[:offset] == 7.0) and torch.all(dst[offset + n * h * pitch:] == 7.0)
