"""The ray set-up of the queue schedule (clearance once per pixel, endpoints
once per VPL or, where the pools hold more VPLs than the frame has pixels,
once per ray) against the per-pixel visibility() of the plain schedule: bit
for bit with the IEEE march, at frame sizes around its 8x4 warp tiles and on
both sides of the endpoint table's rule."""
import numpy as np
import pytest
import torch

from instantradiositytest_b200 import _lib as L
from instantradiositytest_b200.runtime import FrameDriver
from instantradiositytest_b200.workload import Workload

pytestmark = pytest.mark.gpu

BUFS = (L.BUF_DIRECT, L.BUF_NOISY, L.BUF_FILTERED)


def render(wl, frames, **options):
    drv = FrameDriver(wl, gpu_gbuffer=True, gpu_vpls=True, **options)
    for i in range(frames):
        drv.step(i)
    torch.cuda.synchronize()
    assert drv.session.check() == L.IRT_OK
    out = [drv.session.buffer(b, torch.uint8).cpu().numpy() for b in BUFS]
    out += [drv.session.reservoirs_host(d, 2).view(np.uint8) for d in (0, 1)]
    out.append(drv.session.buffer(L.BUF_VPL_ARCHIVE, torch.uint8).cpu().numpy())
    drv.close()
    return out


# (width, height, VPLs): the table holds 7 x VPLs entries (history 4) and is used up to width * height.
@pytest.mark.parametrize("size", [(1, 1, 1), (7, 3, 3), (9, 5, 6), (9, 5, 7), (33, 1, 40), (8, 4, 4), (67, 43, 64),
                                  (67, 43, 600)])
@pytest.mark.parametrize("moved", [False, True])
def test_queue_schedule_equals_plain_schedule(cuda, size, moved):
    w, h, vpls = size
    wl = Workload(0, width=w, height=h, vpl_count=vpls, n_lights=3, seed=5 + moved, room_single_mesh=int(moved))
    want = render(wl, 7, fused=0)
    for got in (render(wl, 7, exact_march=True), render(wl, 7, fused=2)):
        for a, b in zip(got, want):
            assert np.array_equal(a, b)
    wl.close()
