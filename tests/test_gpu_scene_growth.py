"""A scene that grows: an update whose memory cannot be had fails and leaves the
scene as it was, renderable as before and charged as before; later growth of
lights and objects works.  The failing update asks for more lights than any
device holds (2^32 - 1: 400 GB), so its allocation is refused at once and the
light array is never read."""
import ctypes as C

import numpy as np
import pytest
import torch

from instantradiositytest_b200 import _lib as L
from instantradiositytest_b200.runtime import FrameDriver, stream_handle
from instantradiositytest_b200.workload import Workload

pytestmark = pytest.mark.gpu


def rendered(steps, fail_before=None):
    wl = Workload(0, width=96, height=64, sdf_resolution=12)
    drv = FrameDriver(wl, gpu_gbuffer=True, gpu_vpls=True)
    scene, ctx = drv.scene, drv.ctx
    for i in range(steps):
        if i == fail_before:
            _, obj, nodes, lights = wl.frame(i)
            held = L.lib.irt_context_bytes_in_use(ctx.handle)
            status = L.lib.irt_scene_update(scene.handle, L.ptr(obj), len(obj), L.ptr(nodes), len(nodes),
                                            L.ptr(lights), 0xFFFFFFFF, stream_handle())
            assert status == L.IRT_E_CUDA
            assert L.lib.irt_context_bytes_in_use(ctx.handle) == held
            # the previous frame's counts still name what the scene holds
            f, *_, vpls, gt = drv.last
            torch.cuda.synchronize()
            g = L.GBuffer(L.GBUFFER_F32, *(gt[k].data_ptr() for k in ("depth", "normal", "color", "params", "motion")))
            pool = torch.zeros(f.counts[1] * 48, dtype=torch.uint8, device="cuda")
            probe = FrameDriver(wl, gpu_gbuffer=True, gpu_vpls=True)
            probe.session.render(scene, f, g, C.c_void_p(pool.data_ptr()), C.c_void_p(pool.data_ptr()))
            torch.cuda.synchronize()
            assert probe.session.check() == L.IRT_OK
            probe.close()
        drv.step(i)
    torch.cuda.synchronize()
    out = [drv.session.buffer(b, torch.uint8).cpu().numpy() for b in (L.BUF_NOISY, L.BUF_FILTERED)]
    # growth that can be had: more lights alone, then more objects
    big = Workload(0, width=96, height=64, sdf_resolution=12, n_lights=40)
    f, obj, nodes, lights = big.frame(0)
    scene.update(obj, nodes, lights)
    held = L.lib.irt_context_bytes_in_use(ctx.handle)
    scene.update(obj, nodes, lights)
    assert L.lib.irt_context_bytes_in_use(ctx.handle) == held
    torch.cuda.synchronize()
    big.close()
    drv.close()
    wl.close()
    return out


def test_failed_growth_leaves_the_scene_as_it_was(cuda):
    a, b = rendered(4), rendered(4, fail_before=2)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
