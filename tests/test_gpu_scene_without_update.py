"""A frame over a scene that has had no update is refused, in every schedule and
in a batch: the scene has no tables a kernel could read."""
import ctypes as C

import pytest
import torch

from instantradiositytest_b200 import _lib as L
from instantradiositytest_b200.batching import Batch
from instantradiositytest_b200.runtime import Context, Scene, Session, gbuffer_device_alloc, session_desc
from instantradiositytest_b200.workload import Workload

pytestmark = pytest.mark.gpu


def test_frames_over_a_scene_without_update_are_refused(cuda):
    wl = Workload(0, width=32, height=16, sdf_resolution=8)
    ctx = Context()
    scene = Scene(ctx, wl.meshes, wl.atlas, wl.sdf_format)
    f, *_ = wl.frame(0)
    f.counts[0] = f.counts[3] = 0  # what such a scene holds
    _, g = gbuffer_device_alloc(16, 32, L.GBUFFER_F32)
    pool = torch.zeros(f.counts[1] * 48, dtype=torch.uint8, device="cuda")
    p = C.c_void_p(pool.data_ptr())
    for fused in (0, 1, 2):
        s = Session(ctx, session_desc(wl.settings, fused=fused))
        with pytest.raises(L.IrtError, match="no update"):
            s.render(scene, f, g, p, p)
        s.close()
    b = Batch(ctx, wl.settings, [(32, 16)])
    with pytest.raises(L.IrtError, match="no update"):
        b.render([scene], [f], [g], [pool.data_ptr()], [pool.data_ptr()])
    b.close()
    torch.cuda.synchronize()
    scene.close()
    ctx.close()
