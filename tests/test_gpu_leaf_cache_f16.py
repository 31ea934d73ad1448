"""The leaf-order cache over coarse f16 fields: a texel is rounded down by up to
2^-10 of its own value, which near a surface is half a voxel, not the distance.
The queue schedule's IEEE march equals the hierarchy walk bit for bit for rooms
that are one field mesh of 4 to 12 samples an axis (voxels of 3.5 to 0.9 m)."""
import ctypes as C

import pytest
import torch

from instantradiositytest_b200 import _lib as L
from instantradiositytest_b200.runtime import Context, Scene, Session, gbuffer_device_alloc, session_desc
from instantradiositytest_b200.workload import Workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("resolution", [4, 5, 6, 8, 12])
@pytest.mark.parametrize("seed", [3, 8, 21])
def test_coarse_f16_fields(cuda, resolution, seed):
    wl = Workload(0, width=161, height=101, seed=seed, room_single_mesh=1, n_lights=3, vpl_count=64, n_boxes=8,
                  n_spheres=10, sdf_resolution=resolution, sdf_format=L.SDF_F16)
    ctx = Context()
    scene = Scene(ctx, wl.meshes, wl.atlas, wl.sdf_format)
    sessions = [Session(ctx, session_desc(wl.settings, L.GBUFFER_F32, fused=fused, exact_march=True))
                for fused in (1, 0)]
    planes, g = gbuffer_device_alloc(wl.height, wl.width, L.GBUFFER_F32)
    pools = [torch.zeros(64 * 48, dtype=torch.uint8, device="cuda") for _ in range(3)]
    for i in range(6):
        f, objects, nodes, lights = wl.frame(8 * i)
        f.size[2] = i
        f.flags[0] = 1 if i else 0
        f.flags[1] = f.size[3] if i else 0
        # lights and penumbras low enough that rays end lit
        lights["position_strength"][:, 2] = -1.0
        L.check(L.lib.irt_gbuffer_render(ctx.handle, wl.handle, C.byref(f), None, L.GBUFFER_F32, g.depth, g.normal,
                                         g.color, g.params, g.motion, None), ctx.handle, "gbuffer")
        scene.update(objects, nodes, lights)
        cur, prev = pools[i % 2], pools[(i + 1) % 2] if i else pools[2]
        L.check(L.lib.irt_vpl_generate(scene.handle, wl.handle, C.byref(f), C.c_void_p(cur.data_ptr()), None),
                ctx.handle, "vpls")
        for s in sessions:
            s.render(scene, f, g, C.c_void_p(cur.data_ptr()), C.c_void_p(prev.data_ptr()))
        torch.cuda.synchronize()
        for b in (L.BUF_DIRECT, L.BUF_NOISY):
            a, c = (s.buffer(b, torch.uint8) for s in sessions)
            assert torch.equal(a, c), (i, b, int((a != c).sum()))
    for s in sessions:
        assert s.check() == L.IRT_OK
        s.close()
    scene.close()
    ctx.close()
    wl.close()
