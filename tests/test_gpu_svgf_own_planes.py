"""irt_frame_svgf denoises over the planes it is given, whatever the lighting of
the same frame index was given: the lighting's image copied into a session whose
lighting saw the second planes gives the same passes bit for bit."""
import ctypes as C

import numpy as np
import pytest
import torch

from instantradiositytest_b200 import _lib as L
from instantradiositytest_b200.runtime import FrameDriver, gbuffer_to_device, vpls_to_device
from instantradiositytest_b200.workload import Workload

pytestmark = pytest.mark.gpu

BUFS = (L.BUF_TEMPORAL, L.BUF_VARIANCE, L.BUF_MOMENTS, L.BUF_FEEDBACK, L.BUF_FILTERED, L.BUF_PREV_DEPTH,
        L.BUF_PREV_NORMAL)


@pytest.mark.parametrize("formats", [(L.GBUFFER_F32, L.RADIANCE_F32, L.MOMENTS_F32),
                                     (L.GBUFFER_F16, L.RADIANCE_F16, L.MOMENTS_F32),
                                     (L.GBUFFER_PACKED, L.RADIANCE_F16, L.MOMENTS_F16)])
@pytest.mark.parametrize("in_place", [False, True])
def test_svgf_reads_the_planes_it_is_given(cuda, formats, in_place):
    wl = Workload(0, width=96, height=64, sdf_resolution=12)
    a, b = (FrameDriver(wl, gbuffer_format=formats[0], radiance_format=formats[1], moments_format=formats[2])
            for _ in range(2))
    for d in (a, b):
        d.step(0)
    f, obj, nodes, lights, planes, vpls = a.inputs(1)
    # other planes: the objects' materials and half the image's depths and normals of another view
    _, _, _, _, other, _ = a.inputs(9)
    first, g1 = gbuffer_to_device(planes, a.fmt)
    second, g2 = gbuffer_to_device(other, a.fmt)
    pool = vpls_to_device(vpls)
    cur, prev = C.c_void_p(pool.data_ptr()), C.c_void_p(a.prev_vpls.data_ptr())
    for d, g in ((a, g1), (b, g2)):
        d.scene.update(obj, nodes, lights)
        d.session.lighting(d.scene, f, g, cur, prev)
    torch.cuda.synchronize()
    b.session.buffer(L.BUF_NOISY, torch.uint8).copy_(a.session.buffer(L.BUF_NOISY, torch.uint8))
    if in_place:  # the first planes' own memory, edited between the calls
        for k in first:
            first[k].copy_(second[k])
    torch.cuda.synchronize()
    a.session.svgf(f, g1 if in_place else g2)
    b.session.svgf(f, g2)
    torch.cuda.synchronize()
    for w in BUFS:
        assert np.array_equal(a.session.buffer(w, torch.uint8).cpu().numpy(),
                              b.session.buffer(w, torch.uint8).cpu().numpy()), w
    for d in (a, b):
        d.close()
    wl.close()
