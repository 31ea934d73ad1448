"""Frames whose pixel count is no multiple of a vector load (W*H odd) through
the entry points that lay the G-buffer planes out themselves: the host-input
path and the render server.  Every plane must start on an aligned address
whatever the size, and the images must be those of the same frames rendered
from device planes of the caller's."""
import numpy as np
import pytest
import torch

from instantradiositytest_b200 import _lib as L
from instantradiositytest_b200.runtime import Context, FrameDriver, Scene, Session, session_desc
from instantradiositytest_b200.serving import Server
from instantradiositytest_b200.workload import Workload

pytestmark = pytest.mark.gpu

FRAMES = 3


def images(wl, gfmt, rad):
    ref = FrameDriver(wl, gbuffer_format=gfmt, radiance_format=rad, gpu_gbuffer=True, gpu_vpls=True)
    out = []
    for i in range(FRAMES):
        ref.step(i)
        out.append(ref.session.buffer(L.BUF_FILTERED, torch.uint8).cpu().numpy())
    return ref, out


@pytest.mark.parametrize("gfmt,rad", [(L.GBUFFER_F32, L.RADIANCE_F32), (L.GBUFFER_F16, L.RADIANCE_F16)])
@pytest.mark.parametrize("size", [(65, 41), (63, 38)])
def test_host_planes_of_ragged_frames(cuda, gfmt, rad, size):
    wl = Workload(0, width=size[0], height=size[1])
    ctx = Context()
    ref = FrameDriver(wl, ctx=ctx, gbuffer_format=gfmt, radiance_format=rad)
    scene = Scene(ctx, wl.meshes, wl.atlas, wl.sdf_format)
    sess = Session(ctx, session_desc(wl.settings, gfmt, rad))
    keep = []
    for i in range(FRAMES):
        inputs = ref.inputs(i)
        f, obj, nodes, lights, planes, vpls = inputs
        ref.step(i, inputs=inputs)
        g = {k: torch.from_numpy(np.ascontiguousarray(v).view(np.uint8).reshape(-1)).pin_memory()
             for k, v in planes.items()}
        hv = torch.from_numpy(vpls.view(np.uint8)).pin_memory()
        scene.update(obj, nodes, lights)
        sess.render_host(scene, f, L.GBuffer(gfmt, *(g[k].data_ptr() for k in ("depth", "normal", "color", "params",
                                                                              "motion"))), hv)
        keep.append((g, hv))
    sess.host_sync()
    torch.cuda.synchronize()
    for which in (L.BUF_FILTERED, L.BUF_DIRECT):
        assert torch.equal(sess.buffer(which, torch.uint8), ref.session.buffer(which, torch.uint8))
    for h in (sess, scene, ref):
        h.close()
    ctx.close()


@pytest.mark.parametrize("gfmt,rad", [(L.GBUFFER_F32, L.RADIANCE_F32), (L.GBUFFER_F16, L.RADIANCE_F16)])
def test_served_planes_of_ragged_frames(cuda, gfmt, rad):
    wl = Workload(0, width=65, height=41)
    ref, want = images(wl, gfmt, rad)
    server = Server(ref.ctx, 4 << 30, streams=1, frame_rate=0.0, gbuffer_format=gfmt, radiance_format=rad)
    got = server.submit(0, 0.0, FRAMES, wl, capture_frame=FRAMES - 1)
    server.run()
    server.close()
    assert np.array_equal(got, want[-1])
    ref.close()
