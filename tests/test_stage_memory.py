"""Whose memory the stage's device pointers are: only the context's own GPU's (and managed
memory) is read and written by its kernels in place, checked for every kind of pointer
without a GPU; other buffers, as page-locked host memory, go through copies with the
oracle's outputs."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

CHECK = """
#include "caller_memory.h"
int main() {
    struct { cudaMemoryType type; int device, want; } cases[] = {
        {cudaMemoryTypeDevice, 1, 1}, {cudaMemoryTypeDevice, 0, 0},  {cudaMemoryTypeDevice, 2, 0},
        {cudaMemoryTypeHost, 1, 0},   {cudaMemoryTypeHost, 0, 0},    {cudaMemoryTypeUnregistered, 1, 0},
        {cudaMemoryTypeManaged, 1, 1}, {cudaMemoryTypeManaged, 0, 1}};
    for (const auto& c : cases) {
        cudaPointerAttributes a{};
        a.type = c.type;
        a.device = c.device;
        if (ftb::in_place(a, 1) != static_cast<bool>(c.want)) return 1;
    }
    return 0;
}
"""


def test_pointer_kinds(tmp_path):
    gxx, cuda = shutil.which("g++"), "/usr/local/cuda/include"
    if not gxx or not os.path.isdir(cuda):
        pytest.skip("no host C++ compiler or CUDA headers")
    src = tmp_path / "check.cpp"
    src.write_text(CHECK)
    subprocess.run([gxx, "-std=c++17", "-o", str(tmp_path / "check"), str(src), "-I" + cuda,
                    "-I" + os.path.join(ROOT, "fainttrail_b200", "csrc")], check=True)
    subprocess.run([str(tmp_path / "check")], check=True)


@pytest.mark.gpu
@pytest.mark.parametrize("frames_host,out_host", [(True, True), (True, False), (False, True)])
@pytest.mark.parametrize("w,h,pitch", [(64, 33, 64), (67, 17, 70)])
def test_page_locked(device, oracle, frames_host, out_host, w, h, pitch):
    import torch
    rng = np.random.default_rng(w)
    n = 9
    sub = rng.normal(0, 1, (n, h, w)).astype(np.float32)
    t = np.linspace(-0.3, 0.3, n)
    place = lambda a, host: a.pin_memory() if host else a.cuda()  # noqa: E731
    src = torch.full((n, h, pitch), 7.0)
    src[:, :, :w] = torch.from_numpy(sub)
    frames, out = place(src, frames_host), place(torch.full((n, h, pitch), 7.0), out_host)
    torch.cuda.synchronize()
    got = device.stage_dev(frames.data_ptr(), w, h, pitch, n, t, 2.0, out.data_ptr())
    want = oracle.build_stage(sub, t, 2.0)
    assert np.array_equal(out[:, :, :w].cpu().numpy(), want["filtered"], equal_nan=True)
    assert torch.all(out[:, :, w:] == 7.0) and np.array_equal(got["sigma"], want["sigma"])
