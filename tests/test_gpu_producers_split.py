"""Both ways of the CUDA producers: VPL paths with a warp each (up to 8192) and
with a thread each (above) are the same paths bit for bit, and the G-buffer's
per-block primitive lists see what the CPU producer sees at ragged sizes, from
a one-block frame up, in scenes of a few objects and of many."""
import ctypes as C

import numpy as np
import pytest
import torch

from instantradiositytest_b200 import _lib as L
from instantradiositytest_b200.runtime import Context, Scene, gbuffer_device_alloc, stream_handle
from instantradiositytest_b200.workload import Workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("boxes,spheres", [(2, 1), (60, 40)])
def test_shared_and_single_thread_paths_are_the_same(cuda, boxes, spheres):
    wl = Workload(1, width=64, height=40, sdf_resolution=12, n_boxes=boxes, n_spheres=spheres)
    ctx = Context()
    scene = Scene(ctx, wl.meshes, wl.atlas, wl.sdf_format)
    f, obj, nodes, lights = wl.frame(0)
    scene.update(obj, nodes, lights)
    pools = []
    for n in (33, 8192, 8193):
        f.counts[1] = n
        out = torch.zeros(n * 48, dtype=torch.uint8, device="cuda")
        L.check(L.lib.irt_vpl_generate(scene.handle, wl.handle, C.byref(f), C.c_void_p(out.data_ptr()),
                                       stream_handle()), ctx.handle, "vpls")
        pools.append(out.cpu().numpy().view(L.VPL_DTYPE))
    for few, many in ((pools[0], pools[1]), (pools[1], pools[2])):
        n = len(few)
        assert np.array_equal(few["position"], many["position"][:n])
        assert np.array_equal(few["normal"], many["normal"][:n])
        # flux is divided by the path count last: one rounding either side
        a, b = few["flux"].astype(np.float64) * n, many["flux"][:n].astype(np.float64) * len(many)
        assert np.all(np.abs(a - b) <= 2.5e-7 * np.abs(a))
    assert (pools[2]["flux"][:, :3].max(1) > 0).mean() > 0.3
    scene.close()
    ctx.close()
    wl.close()


@pytest.mark.parametrize("size", [(1, 1), (31, 9), (33, 7), (200, 125)])
@pytest.mark.parametrize("boxes,spheres,single", [(2, 1, 1), (14, 9, 0), (100, 60, 1)])
def test_listed_primitives_see_what_the_cpu_sees(cuda, size, boxes, spheres, single):
    wl = Workload(1, width=size[0], height=size[1], sdf_resolution=12, n_boxes=boxes, n_spheres=spheres,
                  room_single_mesh=single)
    ctx = Context()
    for index in (0, 17, 40):
        f, *_ = wl.frame(index)
        c = wl.gbuffer_cpu(f)
        t, g = gbuffer_device_alloc(wl.height, wl.width, L.GBUFFER_F32)
        L.check(L.lib.irt_gbuffer_render(ctx.handle, wl.handle, C.byref(f), None, L.GBUFFER_F32, g.depth, g.normal,
                                         g.color, g.params, g.motion, stream_handle()), ctx.handle, "gbuffer")
        depth = t["depth"].cpu().numpy().view(np.float32).reshape(wl.height, wl.width)
        color = t["color"].cpu().numpy().view(np.float32).reshape(wl.height, wl.width, 4)
        # as the full-size test: depth within 1e-4 and the same material, silhouettes aside
        same = (np.abs(depth - c["depth"]) <= 1e-4) & (color == c["color"]).all(-1)
        assert same.mean() >= 0.99, (index, same.mean())
    ctx.close()
    wl.close()
