"""The G-buffer producer's per-block primitive lists leave nothing visible out,
whatever the projection.  A table of more than 2048 primitives is not listed,
so the same objects with 2100 more out of sight (beyond every far plane) render
without lists: all planes are equal bit for bit.  Perspective, telephoto and
parallel views, mirrored, with a tilted near plane and from far off the origin,
at sizes with ragged blocks.  And the analytic solids in parallel views against
the CPU producer, silhouettes aside."""
import ctypes as C

import numpy as np
import pytest
import torch

from instantradiositytest_b200 import _lib as L
from instantradiositytest_b200 import scene_file as sf
from instantradiositytest_b200.runtime import Context, gbuffer_device_alloc, stream_handle
from instantradiositytest_b200.workload import Workload

pytestmark = pytest.mark.gpu


def look_at(eye, target):
    z = np.asarray(eye, np.float64) - target
    z /= np.linalg.norm(z)
    x = np.cross([0, 0, 1.0], z)
    x /= np.linalg.norm(x)
    m = np.eye(4)
    m[:3, :3] = x, np.cross(z, x), z
    m[:3, 3] = -m[:3, :3] @ eye
    return m


def perspective(fov, aspect, near, far):
    t = 1 / np.tan(fov / 2)
    return np.array([[t / aspect, 0, 0, 0], [0, t, 0, 0], [0, 0, far / (near - far), near * far / (near - far)],
                     [0, 0, -1, 0]])


def parallel(height, aspect, near, far):
    return np.array([[2 / (height * aspect), 0, 0, 0], [0, 2 / height, 0, 0],
                     [0, 0, 1 / (near - far), near / (near - far)], [0, 0, 0, 1]])


def tilted(proj, tilt):
    """The near plane turned: depth also grows with the view-space x and y."""
    out = proj.copy()
    out[2] += tilt * np.array([.3, -.2, 0, 0])
    return out


def frame_of(vp, width, height):
    f = L.Frame()
    f.size[0], f.size[1] = width, height
    for dst, src in ((f.vp, vp), (f.inv_vp, np.linalg.inv(vp)), (f.previous_vp, vp)):
        dst.m[:] = [float(v) for v in src.T.reshape(-1)]
    return f


def render(ctx, wl, f):
    w, h = f.size[0], f.size[1]
    t, g = gbuffer_device_alloc(h, w, L.GBUFFER_F32)
    L.check(L.lib.irt_gbuffer_render(ctx.handle, wl.handle, C.byref(f), None, L.GBUFFER_F32, g.depth, g.normal,
                                     g.color, g.params, g.motion, stream_handle()), ctx.handle, "gbuffer")
    return {k: v.cpu().numpy() for k, v in t.items()}


@pytest.fixture(scope="module", params=[(0.0, 0.0, 0.0), (900.0, -700.0, 300.0)], ids=["origin", "far_off"])
def scenes(request, tmp_path_factory):
    offset = np.array(request.param)
    rng = np.random.default_rng(5)
    visible = []
    for k in range(120):
        q = rng.normal(size=4)
        visible.append(sf.obj(f"o{k}", "cube", f"m{k % 7}", offset + rng.uniform(-6, 6, 3), q / np.linalg.norm(q),
                              float(np.exp(rng.uniform(np.log(.03), np.log(1.2))))))
    hidden = [sf.obj(f"x{k}", "cube", "m0", (3e5 + 4 * k, 0, 0)) for k in range(2100)]
    materials = [sf.material(f"m{k}", rng.uniform(.1, .9, 3)) for k in range(7)]
    paths = []
    for name, objects in (("few", visible), ("many", visible + hidden)):
        scene = sf.Scene([sf.box("cube", (-1, -1, -1), (1, 1, 1), resolution=8)], materials, objects,
                         [sf.point_light("l", offset)],
                         {"position": [float(v) for v in offset + (0, -9, 1)], "rotation": [0.0, 0.0, 0.0, 1.0],
                          "fov_y_radians": .8, "near": .1, "far": 100.0})
        paths.append(sf.write_scene(str(tmp_path_factory.mktemp(name)), scene))
    few, many = (Workload.load(p, width=64, height=40) for p in paths)
    yield offset, few, many
    few.close()
    many.close()


VIEWS = {
    "perspective": lambda a: perspective(.9, a, .1, 1000.0),
    "short_range": lambda a: perspective(1.2, a, 1.0, 40.0),
    "telephoto": lambda a: perspective(.0175, a, .1, 1000.0),
    "parallel_10m": lambda a: parallel(10 / a, a, .1, 60.0),
    "parallel_half_m": lambda a: parallel(.5, a, .1, 1000.0),
    "mirrored": lambda a: np.diag([-1.0, 1, 1, 1]) @ perspective(.9, a, .1, 1000.0),
    "mirrored_parallel": lambda a: np.diag([1.0, -1, 1, 1]) @ parallel(10 / a, a, .1, 60.0),
    "reversed_depth": lambda a: np.array([[1, 0, 0, 0], [0, 1, 0, 0], [0, 0, -1, 1], [0, 0, 0, 1.0]]) @
    perspective(.9, a, .1, 1000.0),
    "tilted_near": lambda a: tilted(perspective(.9, a, .5, 50.0), .4),
}


@pytest.mark.parametrize("view", VIEWS)
@pytest.mark.parametrize("size", [(33, 7), (160, 100), (641, 401), (1281, 721)])
def test_lists_change_no_bit(cuda, scenes, view, size):
    offset, few, many = scenes
    ctx = Context()
    seen = 0
    for eye in ((0, -9, 1), (5, 6, -3)):
        vp = VIEWS[view](size[0] / size[1]) @ look_at(offset + eye, offset + (.2, .1, 0))
        f = frame_of(vp, *size)
        a, b = render(ctx, few, f), render(ctx, many, f)
        for k in a:
            assert np.array_equal(a[k], b[k]), (k, (a[k] != b[k]).reshape(size[1], size[0], -1).any(-1).sum())
        seen += int((a["depth"].view(np.float32) < 1).sum())
    assert seen > 0
    ctx.close()


@pytest.mark.parametrize("size", [(160, 100), (640, 400)])
@pytest.mark.parametrize("boxes,spheres", [(2, 12), (14, 9)])
def test_parallel_views_of_the_room_match_the_cpu(cuda, size, boxes, spheres):
    wl = Workload(1, width=size[0], height=size[1], sdf_resolution=12, n_boxes=boxes, n_spheres=spheres)
    ctx = Context()
    for eye in ((3.5, 0, -3.2), (-1, 4, 3)):
        f = frame_of(parallel(6.0, size[0] / size[1], .05, 30.0) @ look_at(np.array(eye), np.array([0, 0, -4.0])), *size)
        c, g = wl.gbuffer_cpu(f), render(ctx, wl, f)
        color = g["color"].view(np.float32).reshape(size[1], size[0], 4)
        ids = {v: k for k, v in enumerate({tuple(v) for v in c["color"].reshape(-1, 4)})}
        want = np.array([ids[tuple(v)] for v in c["color"].reshape(-1, 4)]).reshape(size[1], size[0])
        got = np.array([ids.get(tuple(v), -1) for v in color.reshape(-1, 4)]).reshape(size[1], size[0])
        padded = np.pad(want, 1, mode="edge")
        near = np.stack([padded[1 + y:1 + y + size[1], 1 + x:1 + x + size[0]] for y in (-1, 0, 1) for x in (-1, 0, 1)])
        inside = (near == want).all(0)  # away from silhouettes and edges of solids
        assert len(ids) > 3 and inside.mean() > .8
        assert np.array_equal(got[inside], want[inside]), int((got != want)[inside].sum())
    ctx.close()
    wl.close()
