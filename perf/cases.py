"""Performance cases of the lighting framework: what a program that uses it
has it do, over the sizes, storage formats and options of its configurations.

Kinds of a case
  frame     one frame of a session whose G-buffer and VPL pool are on the
            device: scene update + lighting + SVGF (irt_render_frame)
  produced  the same with the G-buffer and the VPLs rendered on the device in
            the pass (FrameDriver.step)
  host      a frame whose G-buffer and VPLs come from pinned host memory and
            whose image goes back there (irt_render_frame_host)
  views     one frame of several views of uneven size (BatchDriver.step)
  serve     a run of the render server over a handful of sessions
  svgf      the denoiser alone over a program's own lighting (irt_frame_svgf)
  filter    the allocation-free spatial filter (irt_svgf_spatial_noalloc)

Storage: "f32" (every plane f32), "f16" (the reference's render targets:
f16 G-buffer and radiance, f32 moments and SDF), "mixed" (packed G-buffer,
f16 SDF, radiance and moments).
"""
import ctypes as C
import math

import numpy as np
import torch

from instantradiositytest_b200 import _lib as L
from instantradiositytest_b200.batching import BatchDriver
from instantradiositytest_b200.runtime import (Context, FrameDriver, Scene, Session, gbuffer_device_alloc,
                                               gbuffer_struct, session_desc, stream_handle)
from instantradiositytest_b200.serving import Server
from instantradiositytest_b200.workload import Workload, preset_spec

STORAGE = {  # G-buffer, radiance, moments, SDF texels
    "f32": (L.GBUFFER_F32, L.RADIANCE_F32, L.MOMENTS_F32, L.SDF_F32),
    "f16": (L.GBUFFER_F16, L.RADIANCE_F16, L.MOMENTS_F32, L.SDF_F32),
    "mixed": (L.GBUFFER_PACKED, L.RADIANCE_F16, L.MOMENTS_F16, L.SDF_F16),
}
WARMUP = 5   # frames rendered before the timed ones, so that every history exists
PATH = 4     # camera positions of a frame case, walked forth and back


def _room(kind, width, height, storage, boxes, spheres, res, lights, vpls, single=True, **options):
    return dict(kind=kind, width=width, height=height, storage=storage, boxes=boxes, spheres=spheres, res=res,
                lights=lights, vpls=vpls, single=single, **options)


def listed():
    return [
        # The reference's own GPU-test size, one light, certified-box walls: latency and launches.
        dict(_room("frame", 160, 100, "f32", 4, 2, 64, 1, 100, single=False), name="frame_160x100_f32"),
        # A preview window in the reference's own render-target formats.
        dict(_room("frame", 480, 300, "f16", 8, 5, 64, 4, 512), name="frame_480x300_f16"),
        # A dynamic scene: objects move every frame, so the hierarchy and the scene records change.
        dict(_room("frame", 960, 600, "f32", 14, 9, 64, 8, 1024, moving=True), name="moving_960x600_f32"),
        # The default workload: 24 meshes at 128^3, 8 emitters, 1024 VPLs.
        dict(_room("frame", 1920, 1200, "f32", 14, 9, 128, 8, 1024), name="frame_1920x1200_f32"),
        # The same in the mixed-precision storage.
        dict(_room("frame", 1920, 1200, "mixed", 14, 9, 128, 8, 1024), name="frame_1920x1200_mixed"),
        # A ragged window with the reference's hardware-filtered field sampler.
        dict(_room("frame", 1283, 717, "f32", 10, 7, 96, 5, 600, linear=True), name="frame_1283x717_linear"),
        # The largest session a server is given: a crowded room, more lights than the small-scene table holds.
        dict(_room("frame", 2560, 1600, "mixed", 30, 20, 64, 12, 1024), name="frame_2560x1600_mixed"),
        # A frame with its inputs rendered on the device, as the server and the frame driver run it.
        dict(_room("produced", 1280, 720, "f16", 10, 7, 64, 4, 512), name="produced_1280x720_f16"),
        # A host that keeps its render targets in its own (pinned) memory.
        dict(_room("host", 1920, 1200, "mixed", 14, 9, 64, 8, 1024), name="host_1920x1200_mixed"),
        # Eight views of two scenes in one batch, each frame replayed as a graph.
        dict(_room("views", 1280, 800, "mixed", 12, 8, 64, 6, 512, views=8, scenes=2), name="views_8_mixed"),
        # Four short sessions through the render server.
        dict(_room("serve", 960, 600, "mixed", 8, 6, 64, 4, 512, sessions=4, frames=20), name="serve_4_mixed"),
        # The denoiser alone at full HD in the reference's formats.
        dict(kind="svgf", width=1920, height=1080, storage="f16", iterations=4, name="svgf_1920x1080_f16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame"] * 6 + ["produced", "host", "views", "svgf", "filter"])
    storage = rng.choice(["f32", "f16", "mixed"])
    if kind == "filter":  # at most 512x512 pixels
        return dict(kind=kind, width=_log_int(rng, 64, 512), height=_log_int(rng, 40, 512), storage=storage,
                    iterations=rng.choice([1, 3, 4, 5]))
    width = _log_int(rng, 128, 1920)
    height = max(8, int(width * rng.uniform(0.5, 0.75)))
    if kind == "svgf":
        return dict(kind=kind, width=width, height=height, storage=storage, iterations=rng.choice([1, 3, 4, 5]))
    case = _room(kind, width, height, storage, rng.randint(2, 30), rng.randint(1, 20), rng.choice([32, 48, 64, 96]),
                 rng.randint(1, 12), _log_int(rng, 64, 2048), single=rng.random() < 0.7)
    if kind == "frame":
        pick = rng.random()
        if pick < 0.2:
            case["moving"] = True
        elif pick < 0.4:
            case["storage"], case["linear"] = rng.choice(["f32", "f16"]), True
        elif pick < 0.5:
            case["exact_march"] = True
    if kind == "host":
        case["width"] = max(8, width // 8 * 8)  # render targets' rows come in whole vectors
    if kind == "views":
        case.update(width=min(width, 1280), height=min(height, 800), views=rng.randint(2, 10),
                    scenes=rng.randint(1, 3))
    return case


class _Handles:
    """The framework handles of one program, closed when nothing reads their buffers any more."""

    def __init__(self):
        self.open = []

    def __del__(self):
        try:
            torch.cuda.synchronize()
            while self.open:
                self.open.pop().close()
        except Exception:
            pass


class _Program:
    """What one program holds: its handles, inputs, and tensors over its outputs."""

    def __init__(self):
        self.handles = _Handles()
        self.next = 0

    def keep(self, handle):
        self.handles.open.append(handle)
        return handle


class _Buffer:
    """A session buffer for torch; a tensor over it keeps the session's handles open."""

    def __init__(self, handles, ptr, nbytes):
        self.handles = handles
        self.__cuda_array_interface__ = {"shape": (nbytes,), "typestr": "|u1", "data": (ptr, False), "version": 3,
                                         "strides": None}


def _tensor(handles, where, dtype, shape):
    ptr, nbytes = where
    return torch.as_tensor(_Buffer(handles, ptr, nbytes), device="cuda").view(dtype).reshape(shape)


def _workload(case, seed, width=None, height=None, k=0):
    w, h = width or case["width"], height or case["height"]
    spec = preset_spec(1, seed=(int(seed) * 16 + k) % (1 << 40), width=w, height=h, n_boxes=case["boxes"],
                       n_spheres=case["spheres"], room_single_mesh=int(case["single"]), sdf_resolution=case["res"],
                       sdf_format=STORAGE[case["storage"]][3], n_lights=case["lights"], vpl_count=case["vpls"])
    return Workload(spec)


def _session_views(handles, s, rad, mom, brief=False):
    """A session's outputs, for the frame just rendered, as tensors over its own buffers
    (brief: the images and the picked samples)."""
    h, w = s.h, s.w
    half = torch.float16 if rad == L.RADIANCE_F16 else torch.float32
    moments = s.buffer_ptr(L.BUF_MOMENTS)
    out = {"filtered": _tensor(handles, s.buffer_ptr(L.BUF_FILTERED), half, (h, w, 4)),
           "noisy": _tensor(handles, s.buffer_ptr(L.BUF_NOISY), half, (h, w, 4)),
           "direct": _tensor(handles, s.buffer_ptr(L.BUF_DIRECT), torch.float32, (h, w, 4))}
    if brief:
        del out["noisy"]
    elif mom == L.MOMENTS_F16:  # (mean, deviation) halves and the f32 history length
        out["moments"] = _tensor(handles, moments, torch.float16, (h, w, 4))[..., :2]
        out["age"] = _tensor(handles, moments, torch.float32, (h, w, 2))[..., 1]
    else:
        out["moments"] = _tensor(handles, moments, torch.float32, (h, w, 4))
    for dom, name in ((0, "light"), (1, "vpl")):
        p, n = C.c_void_p(), C.c_uint64()
        L.check(L.lib.irt_session_reservoirs(s.handle, dom, 2, C.byref(p), C.byref(n)), what="reservoirs")
        out[name + "_picked"] = _tensor(handles, (p.value, n.value), torch.int32, (h, w, 8))[..., :4]
        if not brief:
            out[name + "_weights"] = _tensor(handles, (p.value, n.value), torch.float32, (h, w, 8))[..., 4:7]
    return out


def _moved(objects, meshes, k):
    """The scene's objects with every second one shifted along a small circle,
    and the hierarchy over their boxes: what a program uploads when things move."""
    out = objects.copy()
    for i in range(1, len(out), 2):
        m = out["model"][i].reshape(4, 4).astype(np.float64)  # columns
        a = 2.0 * math.pi * (k + i) / 9.0
        m[3, 0] += 0.03 * math.cos(a)
        m[3, 1] += 0.03 * math.sin(a)
        out["previous"][i] = objects["model"][i]
        out["model"][i] = m.reshape(16).astype(np.float32)
        out["inverse"][i] = np.linalg.inv(m).reshape(16).astype(np.float32)
    n = len(out)
    lo, hi = np.zeros((n, 3), np.float32), np.zeros((n, 3), np.float32)
    for i in range(n):
        mesh = meshes[out["info"][i][0]]
        m = out["model"][i].reshape(4, 4).astype(np.float64)
        corners = np.array([[(mesh["lo"], mesh["hi"])[(c >> a) & 1][a] for a in range(3)] + [1.0] for c in range(8)])
        p = (corners @ m)[:, :3]
        lo[i], hi[i] = p.min(0), p.max(0)
    nodes = np.zeros(2 * n - 1, L.NODE_DTYPE)
    L.check(L.lib.irt_build_hierarchy(L.ptr(lo), L.ptr(hi), n, L.ptr(nodes)), what="hierarchy")
    return out, nodes


def _path(case, wl, ctx, scene, st):
    """Frames over PATH camera positions forth and back: per step its uniform,
    scene data, G-buffer and VPL pool, all made on the device."""
    walk = list(range(PATH)) + list(range(PATH - 2, 0, -1))
    data = [wl.frame(p) for p in range(PATH)]
    st.steps = []
    for j, p in enumerate(walk):
        f, objects, nodes, lights = wl.frame(p)
        before = data[walk[j - 1]][0]
        f.previous_vp, f.previous_inv_vp = before.vp, before.inv_vp
        f.size[2] = j
        if case.get("moving"):
            objects, nodes = _moved(objects, wl.meshes, j)
        scene.update(objects, nodes, lights)
        planes, g = gbuffer_device_alloc(wl.height, wl.width, st.formats[0])
        L.check(L.lib.irt_gbuffer_render(ctx.handle, wl.handle, C.byref(f), None, st.formats[0], g.depth, g.normal,
                                         g.color, g.params, g.motion, stream_handle()), ctx.handle, "gbuffer")
        vpls = torch.zeros(f.counts[1] * 48, dtype=torch.uint8, device="cuda")
        L.check(L.lib.irt_vpl_generate(scene.handle, wl.handle, C.byref(f), C.c_void_p(vpls.data_ptr()),
                                       stream_handle()), ctx.handle, "vpls")
        st.steps.append((f, objects, nodes, lights, planes, g, vpls))


def _frame_state(case, seed, st):
    wl = st.keep(_workload(case, seed))
    ctx = st.ctx = st.keep(Context())
    scene = st.scene = st.keep(Scene(ctx, wl.meshes, wl.atlas, wl.sdf_format))
    if case.get("linear"):
        scene.set_field_filter(L.FIELD_LINEAR)
    _path(case, wl, ctx, scene, st)
    s = st.session = st.keep(Session(ctx, session_desc(wl.settings, *st.formats[:2], True, False,
                                                       case.get("exact_march", False), st.formats[2])))
    st.zero = torch.zeros(wl.settings.vpl_count * 48, dtype=torch.uint8, device="cuda")
    if case["kind"] == "host":
        steps = []
        for f, objects, nodes, lights, planes, g, vpls in st.steps:
            pinned = {k: v.cpu().pin_memory() for k, v in planes.items()}
            steps.append((f, objects, nodes, lights, pinned, gbuffer_struct(pinned, st.formats[0]),
                          vpls.cpu().pin_memory()))
        st.steps = steps
        size = wl.width * wl.height * (8 if st.formats[1] == L.RADIANCE_F16 else 16)
        st.images = [torch.zeros(size, dtype=torch.uint8).pin_memory() for _ in range(2)]
        st.handles.images = st.images  # the last image is written when the session closes
    st.outs = [None, None]
    for _ in range(WARMUP):
        run(st)
        st.outs[(st.next - 1) % 2] = _session_views(st.handles, s, *st.formats[1:3])


def prepare(case, seed):
    st = _Program()
    st.kind = case["kind"]
    st.formats = STORAGE[case["storage"]]
    if st.kind in ("svgf", "filter"):
        _denoise_state(case, seed, st)
    elif st.kind == "produced":
        wl = st.keep(_workload(case, seed))
        drv = st.driver = st.keep(FrameDriver(wl, gbuffer_format=st.formats[0], radiance_format=st.formats[1],
                                              moments_format=st.formats[2], gpu_gbuffer=True, gpu_vpls=True))
        st.outs = [None, None]
        for _ in range(WARMUP):
            run(st)
            st.outs[(st.next - 1) % 2] = _session_views(st.handles, drv.session, *st.formats[1:3])
    elif st.kind == "views":
        rooms = [st.keep(_workload(case, seed, k=k)) for k in range(case["scenes"])]
        views = []
        for v in range(case["views"]):
            w = max(64, int(case["width"] * (1.0 - 0.5 * v / case["views"])) // 16 * 16)
            views.append((rooms[v % len(rooms)], 3 * v, (w, max(1, w * case["height"] // case["width"]))))
        ctx = st.keep(Context())
        st.driver = st.keep(BatchDriver(ctx, views, *st.formats[:3]))
        st.outs = [None, None]
        for _ in range(WARMUP + 1):  # both parities' frames run once directly, then as graphs
            run(st)
            st.outs[(st.next - 1) % 2] = {str(v): _session_views(st.handles, st.driver.batch.view(v), *st.formats[1:3],
                                                                 brief=True) for v in range(case["views"])}
    elif st.kind == "serve":
        st.case = dict(case)
        st.rooms = []
        for k in range(case["sessions"]):
            grow = 1.0 + 0.25 * k
            st.rooms.append(st.keep(_workload(case, seed, int(case["width"] * grow) // 8 * 8,
                                              int(case["height"] * grow) // 8 * 8, k)))
        ctx = st.keep(Context())
        st.server = st.keep(Server(ctx, 32 << 30, streams=2, frame_rate=0.0, gbuffer_format=st.formats[0],
                                   radiance_format=st.formats[1], moments_format=st.formats[2]))
    else:
        _frame_state(case, seed, st)
    return st


def run(st):
    n = st.next
    st.next = n + 1
    if st.kind in ("frame", "host"):
        f, objects, nodes, lights, _, g, vpls = st.steps[n % len(st.steps)]
        f.size[2] = n
        f.flags[0] = 1 if n > 0 else 0
        f.flags[1] = f.size[3] if n > 0 else 0
        st.scene.update(objects, nodes, lights)
        if st.kind == "host":
            st.session.render_host(st.scene, f, g, vpls, st.images[n % 2])
        else:
            prev = st.steps[(n - 1) % len(st.steps)][6] if n > 0 else st.zero
            st.session.render(st.scene, f, g, C.c_void_p(vpls.data_ptr()), C.c_void_p(prev.data_ptr()))
        return st.outs[n % 2]
    if st.kind in ("produced", "views"):
        st.driver.step(n)
        return st.outs[n % 2]
    if st.kind == "serve":
        frames = st.case["frames"]
        images = [st.server.submit(k, 0.0, frames, wl, capture_frame=frames - 1) for k, wl in enumerate(st.rooms)]
        st.server.run()
        return [v.view(np.float16 if st.formats[1] == L.RADIANCE_F16 else np.float32) for v in images]
    if st.kind == "svgf":
        f, g = st.frames[n % 2]
        f.size[2] = n
        f.flags[0] = 1 if n > 0 else 0
        f.flags[1] = f.size[3] if n > 0 else 0
        st.session.svgf(f, g)
        return st.outs[n % 2]
    f, g = st.frames[0]
    err = C.create_string_buffer(256)
    status = L.lib.irt_svgf_spatial_noalloc(C.byref(f), C.byref(g), st.formats[1], st.formats[2], st.iterations,
                                            st.args[0], st.args[1], st.args[2], st.args[3], stream_handle(), err, 256)
    if status != L.IRT_OK:
        raise RuntimeError(err.value.decode())
    return st.outs


# ---------------------------------------------------------------- the denoiser's own inputs
def _camera(seed, width, height, step):
    """vp, inverse and eye of a camera in a 10 m room, in f64 (column-major 4x4 as rows of columns)."""
    a = 0.02 * step + 0.3 * (seed % 17)
    eye = np.array([3.6 * math.cos(a), 3.6 * math.sin(a), -3.2])
    fwd = np.array([0.0, 0.0, -4.0]) - eye
    fwd /= np.linalg.norm(fwd)
    right = np.cross(fwd, [0.0, 0.0, 1.0])
    right /= np.linalg.norm(right)
    up = np.cross(right, fwd)
    view = np.eye(4)
    view[0, :3], view[1, :3], view[2, :3] = right, up, -fwd
    view[:3, 3] = -view[:3, :3] @ eye
    near, far, t = 0.1, 1000.0, 1.0 / math.tan(0.45)
    proj = np.zeros((4, 4))
    proj[0, 0], proj[1, 1] = t * height / width, t
    proj[2, 2], proj[2, 3], proj[3, 2] = far / (near - far), near * far / (near - far), -1.0
    vp = proj @ view
    return vp, np.linalg.inv(vp), eye


def _planes(seed, width, height, step):
    """G-buffer planes (f64 tensors on the device) of a room with spheres seen at a step of the camera path."""
    vp, inv, eye = _camera(seed, width, height, step)
    back = _camera(seed, width, height, 1 - step)
    dev = dict(device="cuda", dtype=torch.float64)
    ys, xs = torch.meshgrid(torch.arange(height, **dev), torch.arange(width, **dev), indexing="ij")
    ndc = torch.stack([(xs + .5) / width * 2 - 1, 1 - (ys + .5) / height * 2, torch.ones_like(xs), torch.ones_like(xs)], -1)
    far = ndc @ torch.tensor(inv.T, **dev)
    o = torch.tensor(eye, **dev)
    d = far[..., :3] / far[..., 3:] - o
    d = d / d.norm(dim=-1, keepdim=True)
    best = torch.full_like(xs, 1e30)
    normal = torch.zeros(height, width, 3, **dev)
    colour = torch.zeros(height, width, 3, **dev)
    params = torch.zeros(height, width, 2, **dev)
    rng = np.random.RandomState(seed % (1 << 31))
    for axis in range(3):
        for side in (-1.0, 1.0):
            if axis == 2 and side > 0:
                continue  # no ceiling: the sky is background
            t = (5.0 * side - o[axis]) / d[..., axis]
            hit = (t > 0) & (t < best) & ((o + d * t[..., None]).abs().amax(-1) <= 5.0 + 1e-9)
            best = torch.where(hit, t, best)
            nrm = torch.zeros(3, **dev)
            nrm[axis] = -side
            normal[hit] = nrm
            colour[hit] = torch.tensor(rng.uniform(.2, .9, 3), **dev)
            params[hit] = torch.tensor([1.0, 0.0], **dev)
    for _ in range(12):
        c = torch.tensor(np.append(rng.uniform(-4, 4, 2), -4.6), **dev)
        r = rng.uniform(.3, .9)
        tint, rough = rng.uniform(.2, .9, 3), rng.uniform(.1, 1.0)
        oc = o - c
        b = (d * oc).sum(-1)
        disc = b * b - (oc @ oc - r * r)
        t = -b - disc.clamp(min=0).sqrt()
        hit = (disc > 0) & (t > 0) & (t < best)
        best = torch.where(hit, t, best)
        normal[hit] = ((o + d * t[..., None] - c) / r)[hit]
        colour[hit] = torch.tensor(tint, **dev)
        params[hit] = torch.tensor([rough, 0.0], **dev)
    seen = best < 1e29
    p = o + d * torch.where(seen, best, torch.ones_like(best))[..., None]
    p1 = torch.cat([p, torch.ones_like(best)[..., None]], -1)
    clip, old = p1 @ torch.tensor(vp.T, **dev), p1 @ torch.tensor(back[0].T, **dev)
    depth = torch.where(seen, clip[..., 2] / clip[..., 3], torch.ones_like(best))
    motion = (clip[..., :2] / clip[..., 3:] - old[..., :2] / old[..., 3:]) * torch.tensor([.5, -.5], **dev)
    motion = torch.where(seen[..., None], motion, torch.zeros_like(motion))
    return depth, normal, colour, params, motion, seen


def _stored(case, seed, step):
    """The planes as the case's storage holds them: (device planes, their values in f64)."""
    fmt = STORAGE[case["storage"]][0]
    depth, normal, colour, params, motion, seen = _planes(seed, case["width"], case["height"], step)
    alpha = seen.double()[..., None]
    depth = depth.float()
    n4, c4 = torch.cat([normal, alpha], -1), torch.cat([colour, alpha], -1)
    if fmt == L.GBUFFER_PACKED:
        s = normal.abs().sum(-1, keepdim=True).clamp(min=1e-30)
        uv = normal[..., :2] / s
        fold = (1 - uv.flip(-1).abs()) * torch.where(uv >= 0, 1.0, -1.0)
        uv = torch.where(normal[..., 2:] < 0, fold, uv)
        q = (uv.clamp(-1, 1) * 32767).round().to(torch.int64)
        pn = ((q[..., 0] & 0xffff) | ((q[..., 1] & 0xffff) << 16))
        qc = (c4.clamp(0, 1) * 255).round().to(torch.int64)
        pc = qc[..., 0] | (qc[..., 1] << 8) | (qc[..., 2] << 16) | (qc[..., 3] << 24)
        low = lambda v: torch.where(v >= 1 << 31, v - (1 << 32), v).to(torch.int32)  # noqa: E731
        planes = dict(depth=depth, normal=low(pn), color=low(pc), params=params.half(), motion=motion.half())
        u, v = (q[..., 0].double() / 32767).clamp(min=-1), (q[..., 1].double() / 32767).clamp(min=-1)
        z = 1 - u.abs() - v.abs()
        t = (-z).clamp(min=0)
        u, v = torch.where(u >= 0, u - t, u + t), torch.where(v >= 0, v - t, v + t)
        back = torch.stack([u, v, z], -1)
        values = (depth.double(), back / back.norm(dim=-1, keepdim=True), qc[..., :3].double() / 255)
    else:
        kind = torch.float16 if fmt == L.GBUFFER_F16 else torch.float32
        planes = dict(depth=depth, normal=n4.to(kind), color=c4.to(kind), params=params.to(kind), motion=motion.to(kind))
        values = (depth.double(), planes["normal"].double()[..., :3], planes["color"].double()[..., :3])
    values = values + (planes["params"].double(), planes["motion"].double())
    return {k: v.contiguous().reshape(-1).view(torch.uint8) for k, v in planes.items()}, values


def _noise(case, seed):
    """A noisy HDR lighting image as a path tracer leaves it: most samples near zero, some bright."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))
    size = (case["height"], case["width"], 1)
    bright = torch.rand(size, generator=g, device="cuda") < 0.35
    v = bright * torch.rand(size, generator=g, device="cuda") * 4.0 + 0.05
    tint = torch.tensor([1.0, 0.8, 0.6], device="cuda")
    img = torch.cat([v * tint, torch.ones(size, device="cuda")], -1)
    return img.half() if STORAGE[case["storage"]][1] == L.RADIANCE_F16 else img


def _frame_uniform(case, seed, step):
    f = L.Frame()
    vp, inv, eye = _camera(seed, case["width"], case["height"], step)
    old_vp, old_inv, _ = _camera(seed, case["width"], case["height"], 1 - step)
    for name, m in (("vp", vp), ("inv_vp", inv), ("previous_vp", old_vp), ("previous_inv_vp", old_inv)):
        getattr(f, name).m[:] = m.T.reshape(16).astype(np.float32).tolist()
    f.camera[:] = [float(v) for v in eye] + [1.0]
    f.size[:] = [case["width"], case["height"], step, 1]
    s = _settings(case)
    f.temporal[:] = [s.temporal_history_weight, s.depth_threshold, s.normal_threshold, float(s.temporal_max_history)]
    return f


def _settings(case):
    s = L.Settings()
    L.lib.irt_settings_default(C.byref(s))
    s.render_width, s.render_height, s.svgf_iterations = case["width"], case["height"], case["iterations"]
    return s


def _temporal_inputs(case, seed):
    """Moments of a young history for the spatial filter alone: (image, E[l], E[l^2] or the deviation, age), f64."""
    img = _noise(case, seed).double()[..., :3]
    lum = img @ torch.tensor([.2126, .7152, .0722], device="cuda", dtype=torch.float64)
    g = torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62) + 1)
    age = torch.randint(1, 9, lum.shape, generator=g, device="cuda").double()
    mean = (lum * .8 + .1).float().double()
    dev = (lum * .3 + .05).float().double()
    return img, mean, dev, age


def _denoise_state(case, seed, st):
    st.iterations = case["iterations"]
    gfmt, rad, mom, _ = st.formats
    st.planes = [_stored(case, seed, k)[0] for k in range(2 if st.kind == "svgf" else 1)]
    st.frames = [(_frame_uniform(case, seed, k), gbuffer_struct(p, gfmt)) for k, p in enumerate(st.planes)]
    noisy = _noise(case, seed)
    if st.kind == "svgf":
        ctx = st.keep(Context())
        s = st.session = st.keep(Session(ctx, session_desc(_settings(case), gfmt, rad, moments_format=mom)))
        target = s.buffer(L.BUF_NOISY, torch.uint8)
        target.copy_(noisy.reshape(-1).view(torch.uint8))
        st.outs = [None, None]
        run(st)  # the first frame has no history
        for k in (0, 1):
            kind = torch.float16 if rad == L.RADIANCE_F16 else torch.float32
            st.outs[k] = {"filtered": _tensor(st.handles, s.buffer_ptr(L.BUF_FILTERED), kind, (s.h, s.w, 4))}
        return
    img, mean, dev, age = _temporal_inputs(case, seed)
    h, w = age.shape
    sigma = dev.to(noisy.dtype)[..., None]
    image = torch.cat([noisy[..., :3], sigma], -1).contiguous()
    if mom == L.MOMENTS_F16:
        moments = torch.empty(h, w, 2, dtype=torch.float32, device="cuda")
        moments.view(torch.float16).reshape(h, w, 4)[..., :2] = torch.stack([mean, dev], -1).half()
        moments[..., 1] = age
    else:
        moments = torch.stack([mean, dev * dev + mean * mean, age, age * 0], -1).float().contiguous()
    outs = [torch.zeros_like(image) for _ in range(2)]
    st.buffers = (image, moments)
    st.args = [C.c_void_p(t.data_ptr()) for t in (image, moments, *outs)]
    st.outs = {"filtered": outs[0], "feedback": outs[1]}


# ---------------------------------------------------------------- the denoiser in 64 bits
class _Exact:
    """svgf_temporal, svgf_variance and svgf_atrous over f64 tensors."""

    def __init__(self, case, seed, step):
        self.h, self.w = case["height"], case["width"]
        self.depth, self.normal, self.colour, self.params, self.motion = _stored(case, seed, step)[1]
        f = _frame_uniform(case, seed, step)
        self.f = f
        dev = dict(device="cuda", dtype=torch.float64)
        inv = torch.tensor(list(f.inv_vp.m), **dev).reshape(4, 4)  # rows are columns
        self.ys, self.xs = torch.meshgrid(torch.arange(self.h, device="cuda"), torch.arange(self.w, device="cuda"),
                                          indexing="ij")
        p = torch.stack([(self.xs + .5) / self.w * 2 - 1, 1 - (self.ys + .5) / self.h * 2, self.depth,
                         torch.ones_like(self.depth)], -1).to(torch.float64) @ inv
        self.position = p[..., :3] / p[..., 3:]
        self.camera = torch.tensor(list(f.camera)[:3], **dev)
        self.distance = (self.position - self.camera).norm(dim=-1)
        self.scale = self.distance / self.h
        self.lum = torch.tensor([.2126, .7152, .0722], **dev)

    def tap(self, dx, dy):
        y, x = self.ys + dy, self.xs + dx
        inside = (y >= 0) & (x >= 0) & (y < self.h) & (x < self.w)
        return y.clamp(0, self.h - 1), x.clamp(0, self.w - 1), inside

    def geometry(self, y, x, inside, stride):
        wn = (self.normal * self.normal[y, x]).sum(-1).clamp(min=0) ** 64
        tol = (self.scale * stride * .5).clamp(min=.0001)
        wz = torch.exp(-((self.position[y, x] - self.position) * self.normal).sum(-1).abs() / tol)
        wc = torch.exp(-(self.colour - self.colour[y, x]).norm(dim=-1) * 8
                       - (self.params - self.params[y, x]).norm(dim=-1) * 8)
        return torch.where(inside & (self.depth[y, x] < 1), wn * wz * wc, torch.zeros_like(wn))

    def temporal(self, noisy, old):
        """`old`: (the previous frame's _Exact, radiance, moment 1, variance or moment 2, age), or None."""
        l = noisy @ self.lum
        one = torch.ones_like(l)
        if old is None:
            return noisy, torch.zeros_like(l), l, l * l, one
        was, radiance, om1, om2, oage = old
        px = ((self.xs + .5) / self.w - self.motion[..., 0]) * self.w - .5
        py = ((self.ys + .5) / self.h - self.motion[..., 1]) * self.h - .5
        bx, by = px.floor(), py.floor()
        fx, fy = px - bx, py - by
        total, hist = torch.zeros_like(l), torch.zeros_like(noisy)
        m1, m2, length = torch.zeros_like(l), torch.zeros_like(l), torch.zeros_like(l)
        reach = self.f.temporal[1] * self.distance.clamp(min=1)
        for yy in (0, 1):
            for xx in (0, 1):
                y, x = (by + yy).long(), (bx + xx).long()
                ok = (y >= 0) & (x >= 0) & (y < self.h) & (x < self.w) & (self.depth < 1)
                y, x = y.clamp(0, self.h - 1), x.clamp(0, self.w - 1)
                ok &= was.depth[y, x] < 1
                ok &= (self.position - was.position[y, x]).norm(dim=-1) < reach
                ok &= (self.normal * was.normal[y, x]).sum(-1) > self.f.temporal[2]
                w = (fx if xx else 1 - fx) * (fy if yy else 1 - fy) * ok * (oage[y, x] > 0)
                hist += radiance[y, x] * w[..., None]
                m1, m2, length, total = m1 + om1[y, x] * w, m2 + om2[y, x] * w, length + oage[y, x] * w, total + w
        ok = total > .001
        t = torch.where(ok, total, one)
        hist, m1, m2 = hist / t[..., None], m1 / t, m2 / t
        age = (length / t + 1).clamp(max=self.f.temporal[3])
        lo, hi = torch.full_like(l, 1e20), torch.zeros_like(l)
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                y, x, _ = self.tap(dx, dy)
                near = self.geometry(y, x, torch.ones_like(ok), 1.0) > .01
                v = l[y, x]
                lo, hi = torch.where(near, torch.minimum(lo, v), lo), torch.where(near, torch.maximum(hi, v), hi)
        lh = hist @ self.lum
        clamped = torch.minimum(torch.maximum(lh, lo * .5), hi * 1.5 + .001)
        hist = hist * (clamped / lh.clamp(min=.000001))[..., None]
        alpha = (1 / age).clamp(min=1 - self.f.temporal[0])
        beta = (1 / age).clamp(min=.2)
        res = torch.where(ok[..., None], hist * (1 - alpha[..., None]) + noisy * alpha[..., None], noisy)
        m1, m2 = torch.where(ok, m1 * (1 - beta) + l * beta, l), torch.where(ok, m2 * (1 - beta) + l * l * beta, l * l)
        return res, (m2 - m1 * m1).clamp(min=0).sqrt(), m1, m2, torch.where(ok, age, one)

    def variance(self, sigma, m1, m2, age):
        s0, s1, total = torch.zeros_like(m1), torch.zeros_like(m1), torch.zeros_like(m1)
        for dy in range(-3, 4):
            for dx in range(-3, 4):
                y, x, inside = self.tap(dx, dy)
                w = self.geometry(y, x, inside, 1.0)
                s0, s1, total = s0 + m1[y, x] * w, s1 + m2[y, x] * w, total + w
        n = total.clamp(min=.00001)
        young = (((s1 / n - (s0 / n) ** 2).clamp(min=0)) * 4 / age.clamp(min=1)).sqrt()
        return torch.where((age < 4) & (self.depth < 1), young, sigma).clamp(max=65000)

    def atrous(self, img, sigma, step):
        var = torch.zeros_like(sigma)
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                y, x, _ = self.tap(dx, dy)
                var += sigma[y, x] ** 2 * (2 - abs(dx)) * (2 - abs(dy))
        phi = 4 * (var / 16).sqrt() + .0001
        l = img @ self.lum
        total, v, acc = torch.zeros_like(l), torch.zeros_like(l), torch.zeros_like(img)
        kern = (1 / 6, 2 / 3, 1.0, 2 / 3, 1 / 6)
        for dy in range(-2, 3):
            for dx in range(-2, 3):
                y, x, inside = self.tap(dx * step, dy * step)
                w = self.geometry(y, x, inside, float(step)) * kern[dx + 2] * kern[dy + 2]
                w = w * torch.exp(-(l[y, x] - l).abs() / phi)
                acc, total, v = acc + img[y, x] * w[..., None], total + w, v + sigma[y, x] ** 2 * w * w
        n = total.clamp(min=.00001)
        sky = self.depth >= 1
        return (torch.where(sky[..., None], img, acc / n[..., None]),
                torch.where(sky, sigma, (v.sqrt() / n).clamp(max=65000)))


def exact(case, seed):
    """The denoiser's image in 64 bits.  A rendered frame has no such value:
    which light or VPL a pixel keeps is decided by comparing random draws
    with f32 sums, so another precision is another image."""
    if case["kind"] not in ("svgf", "filter"):
        return None
    whole = lambda img, sigma: torch.cat([img, sigma[..., None]], -1)  # noqa: E731
    noisy = _noise(case, seed).double()[..., :3]
    if case["kind"] == "filter":
        e = _Exact(case, seed, 0)
        img, mean, dev, age = _temporal_inputs(case, seed)
        kind = torch.float16 if STORAGE[case["storage"]][1] == L.RADIANCE_F16 else torch.float32
        sigma = dev.to(kind).double()
        if STORAGE[case["storage"]][2] == L.MOMENTS_F16:
            mean, dev = mean.half().double(), dev.half().double()
        sigma = e.variance(sigma, mean, dev * dev + mean * mean, age)
        first = None
        for i in range(case["iterations"]):
            img, sigma = e.atrous(img, sigma, 1 << i)
            first = first if first is not None else whole(img, sigma)
        return {"filtered": whole(img, sigma), "feedback": first}
    old = None
    for step in (0, 1):
        e = _Exact(case, seed, step)
        img, sigma, m1, m2, age = e.temporal(noisy, old)
        sigma = e.variance(sigma, m1, m2, age)
        for i in range(case["iterations"] if step else 1):
            img, sigma = e.atrous(img, sigma, 1 << i)
        old = (e, img, m1, m2, age)
    return {"filtered": whole(img, sigma)}


def work(case):
    """Bytes: every input plane and history record of a pixel read once and
    every output and new history record written once.  Operations: per pixel
    the candidate and reuse evaluations, the shadow marches (about 48 distance
    queries in a furnished room) and the filter's taps."""
    gb, rad, mom, _ = STORAGE[case["storage"]]
    plane = {L.GBUFFER_F32: 52, L.GBUFFER_F16: 28, L.GBUFFER_PACKED: 20}[gb]
    old = {L.GBUFFER_F32: 20, L.GBUFFER_F16: 12, L.GBUFFER_PACKED: 8}[gb]
    texel = 8 if rad == L.RADIANCE_F16 else 16
    moment = 8 if mom == L.MOMENTS_F16 else 16
    svgf = plane + 2 * old + texel + 2 * texel + 2 * moment + texel  # noisy, feedback in and out, moments, image
    frame = svgf + 2 * 32 * 2 + 16 + texel                           # reservoirs in and out, direct, noisy
    if case["kind"] == "filter":
        pixels, per, flops = case["width"] * case["height"], plane + moment + 3 * texel, 40 * 25 * case["iterations"]
    elif case["kind"] == "svgf":
        pixels, per, flops = case["width"] * case["height"], svgf, 40 * (25 * case["iterations"] + 15)
    else:
        per, flops = frame, 40 * 115 + 30 * 90 + 5800
        pixels = case["width"] * case["height"]
        if case["kind"] == "views":
            pixels = sum((w := max(64, int(case["width"] * (1.0 - 0.5 * v / case["views"])) // 16 * 16))
                         * max(1, w * case["height"] // case["width"]) for v in range(case["views"]))
        elif case["kind"] == "serve":
            pixels = case["frames"] * sum(int(case["width"] * g) // 8 * 8 * (int(case["height"] * g) // 8 * 8)
                                          for g in (1.0 + 0.25 * k for k in range(case["sessions"])))
    return {"bytes": float(pixels * per), "flops": float(pixels * flops)}
