"""Scenes and sessions made and used on a non-blocking stream at once: the
zero-fill of their memory has to be over before the first upload or kernel on
a stream that does not wait for the default one."""
import numpy as np
import pytest
import torch

from instantradiositytest_b200 import _lib as L
from instantradiositytest_b200.runtime import FrameDriver
from instantradiositytest_b200.workload import Workload

pytestmark = pytest.mark.gpu

BUFS = (L.BUF_DIRECT, L.BUF_NOISY, L.BUF_FILTERED, L.BUF_MOMENTS)


def first_frames(wl):
    drv = FrameDriver(wl, gpu_gbuffer=True, gpu_vpls=True)
    for i in range(2):
        drv.step(i)
    torch.cuda.current_stream().synchronize()
    out = [drv.session.buffer(b, torch.uint8).cpu().numpy() for b in BUFS]
    assert drv.session.check() == L.IRT_OK
    drv.close()
    return out


def test_first_frames_on_a_stream_of_their_own(cuda):
    wl = Workload(1, width=640, height=400, sdf_resolution=32, vpl_count=256)
    want = first_frames(wl)
    for _ in range(6):
        with torch.cuda.stream(torch.cuda.Stream()):
            got = first_frames(wl)
        for a, b in zip(got, want):
            assert np.array_equal(a, b)
    wl.close()
