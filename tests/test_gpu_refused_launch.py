"""A launch the device refuses is reported by the call that made it and by no
later one: the allocation-free filter of a frame taller than a grid has rows
fails, the next producer and frame succeed."""
import ctypes as C

import pytest
import torch

from instantradiositytest_b200 import _lib as L
from instantradiositytest_b200.runtime import FrameDriver, gbuffer_device_alloc, stream_handle
from instantradiositytest_b200.workload import Workload

pytestmark = pytest.mark.gpu


def test_a_refused_launch_is_reported_once(cuda):
    wl = Workload(0, width=64, height=40, sdf_resolution=8)
    drv = FrameDriver(wl, gpu_gbuffer=True, gpu_vpls=True)
    drv.step(0)
    f = L.Frame()
    f.size[0], f.size[1] = 1, 70000
    t, g = gbuffer_device_alloc(70000, 1, L.GBUFFER_F32)
    for v in t.values():
        v.zero_()
    image = torch.zeros(70000 * 16, dtype=torch.uint8, device="cuda")
    p = image.data_ptr()
    out = torch.zeros_like(image)
    err = C.create_string_buffer(256)
    status = L.lib.irt_svgf_spatial_noalloc(C.byref(f), C.byref(g), L.RADIANCE_F32, L.MOMENTS_F32, 1, p, p,
                                            out.data_ptr(), None, stream_handle(), err, 256)
    assert status == L.IRT_E_CUDA and b"invalid" in err.value
    drv.step(1)
    torch.cuda.synchronize()
    assert drv.session.check() == L.IRT_OK
    drv.close()
    wl.close()
