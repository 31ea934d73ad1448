"""The leaf-order cache against the plain hierarchy walk: the queue schedule's
IEEE march (which visits a cell's objects in the cache's order and stops at
its bounds) equals the per-entry-point schedule (which walks the hierarchy)
bit for bit — with fewer objects than a cell's 8 entries, with more, above
the 256 objects up to which bounds are object distances, for f16 fields and
the filtered sampler, with objects that move, and far from the origin, where
the f32 error of positions and distances is hundreds of times larger."""
import ctypes as C
import math

import numpy as np
import pytest
import torch

from instantradiositytest_b200 import _lib as L
from instantradiositytest_b200.runtime import Context, Scene, Session, gbuffer_device_alloc, session_desc
from instantradiositytest_b200.workload import Workload

pytestmark = pytest.mark.gpu


def boxes_of(objects, meshes):
    """World boxes of the objects' SDF bounds, and the hierarchy over them."""
    n = len(objects)
    lo, hi = np.zeros((n, 3), np.float32), np.zeros((n, 3), np.float32)
    for i in range(n):
        mesh = meshes[objects["info"][i][0]]
        m = objects["model"][i].reshape(4, 4).astype(np.float64)
        pts = np.array([[(mesh["lo"], mesh["hi"])[(c >> a) & 1][a] for a in range(3)] + [1.0] for c in range(8)]) @ m
        lo[i], hi[i] = np.nextafter(pts[:, :3].min(0).astype(np.float32), -np.inf), np.nextafter(
            pts[:, :3].max(0).astype(np.float32), np.inf)
    nodes = np.zeros(2 * n - 1, L.NODE_DTYPE)
    L.check(L.lib.irt_build_hierarchy(L.ptr(lo), L.ptr(hi), n, L.ptr(nodes)), what="hierarchy")
    return nodes


def moved(objects, k):
    out = objects.copy()
    for i in range(1, len(out), 2):
        m = out["model"][i].reshape(4, 4).astype(np.float64)
        m[3, 0] += 0.05 * math.cos(k + i)
        m[3, 1] += 0.05 * math.sin(k + i)
        out["model"][i] = m.reshape(16)
        out["inverse"][i] = np.linalg.inv(m).reshape(16)
    return out


def shift(f, objects, lights, by):
    """The same frame with the world moved: vp' = vp T(-by), inverse T(by) inv."""
    t = np.eye(4)
    t[:3, 3] = by
    for vp, inv in (("vp", "inv_vp"), ("previous_vp", "previous_inv_vp")):
        m = np.array(getattr(f, vp).m, np.float64).reshape(4, 4).T @ np.linalg.inv(t)
        n = t @ np.array(getattr(f, inv).m, np.float64).reshape(4, 4).T
        getattr(f, vp).m[:] = m.T.reshape(16).astype(np.float32).tolist()
        getattr(f, inv).m[:] = n.T.reshape(16).astype(np.float32).tolist()
    for a in range(3):
        f.camera[a] += by[a]
    objects, lights = objects.copy(), lights.copy()
    for o in objects:
        m = t @ o["model"].reshape(4, 4).T.astype(np.float64)
        o["model"] = o["previous"] = m.T.reshape(16)
        o["inverse"] = np.linalg.inv(m).T.reshape(16)
    lights["position_strength"][:, :3] += np.float32(by)
    return objects, lights


CASES = {
    "few": dict(n_boxes=1, n_spheres=1),
    "room": dict(n_boxes=9, n_spheres=6, sdf_resolution=32),
    "f16": dict(n_boxes=9, n_spheres=6, sdf_resolution=24, sdf_format=L.SDF_F16),
    "linear": dict(n_boxes=9, n_spheres=6, sdf_resolution=24),
    "moving": dict(n_boxes=9, n_spheres=6, sdf_resolution=24),
    "far": dict(n_boxes=9, n_spheres=6, sdf_resolution=24),
    "many": dict(n_boxes=200, n_spheres=90, sdf_resolution=12),
}


@pytest.mark.parametrize("name", list(CASES))
def test_cached_march_equals_hierarchy_walk(cuda, name):
    wl = Workload(0, width=97, height=61, seed=3, room_single_mesh=1, n_lights=3, vpl_count=40, **CASES[name])
    ctx = Context()
    scene = Scene(ctx, wl.meshes, wl.atlas, wl.sdf_format)
    if name == "linear":
        scene.set_field_filter(L.FIELD_LINEAR)
    sessions = [Session(ctx, session_desc(wl.settings, L.GBUFFER_F32, fused=fused, exact_march=True))
                for fused in (1, 0)]
    planes, g = gbuffer_device_alloc(wl.height, wl.width, L.GBUFFER_F32)
    pools = [torch.zeros(40 * 48, dtype=torch.uint8, device="cuda") for _ in range(3)]
    for i in range(4):
        f, objects, nodes, lights = wl.frame(i)
        if name == "moving":
            objects = moved(objects, i)
            nodes = boxes_of(objects, wl.meshes)
        L.check(L.lib.irt_gbuffer_render(ctx.handle, wl.handle, C.byref(f), None, L.GBUFFER_F32, g.depth, g.normal,
                                         g.color, g.params, g.motion, None), ctx.handle, "gbuffer")
        scene.update(objects, nodes, lights)
        cur, prev = pools[i % 2], pools[(i + 1) % 2] if i else pools[2]
        L.check(L.lib.irt_vpl_generate(scene.handle, wl.handle, C.byref(f), C.c_void_p(cur.data_ptr()), None),
                ctx.handle, "vpls")
        torch.cuda.synchronize()
        if name == "far":
            by = (700.0, -300.0, 200.0)
            objects, lights = shift(f, objects, lights, by)
            scene.update(objects, boxes_of(objects, wl.meshes), lights)
            pool = cur.view(torch.float32).reshape(-1, 12)
            pool[:, :3] += torch.tensor(by, device="cuda")
            torch.cuda.synchronize()
        for s in sessions:
            s.render(scene, f, g, C.c_void_p(cur.data_ptr()), C.c_void_p(prev.data_ptr()))
        torch.cuda.synchronize()
        for s in sessions:
            assert s.check() == L.IRT_OK
        for b in (L.BUF_DIRECT, L.BUF_NOISY):
            a, c = (s.buffer(b, torch.uint8) for s in sessions)
            assert torch.equal(a, c), (name, i, b)
        assert sessions[0].image_host(L.BUF_DIRECT).max() > 0
    for s in sessions:
        s.close()
    scene.close()
    ctx.close()
    wl.close()
