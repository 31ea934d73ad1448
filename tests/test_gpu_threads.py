"""Host threads of one process render scenes of very different object counts on
one device in turn: no thread's launches depend on the shared-memory limits
another thread's scene needs, and every image equals the thread's own run
alone.  Single frames in each field sampler's build, and batched views."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest
import torch

from instantradiositytest_b200 import _lib as L
from instantradiositytest_b200.batching import BatchDriver
from instantradiositytest_b200.runtime import Context, FrameDriver
from instantradiositytest_b200.workload import Workload, preset_spec

pytestmark = pytest.mark.gpu

FRAMES = 3
BUFS = (L.BUF_NOISY, L.BUF_FILTERED)


def room(objects, preset):
    return Workload(preset_spec(preset, seed=objects, width=96, height=64, sdf_resolution=8,
                                n_boxes=objects // 2, n_spheres=objects - objects // 2))


def images(session):
    torch.cuda.synchronize()
    return [session.buffer(b, torch.uint8).cpu().numpy() for b in BUFS]


class Single:
    def __init__(self, objects, preset, formats, linear):
        self.driver = FrameDriver(room(objects, preset), gbuffer_format=formats[0], radiance_format=formats[1],
                                  moments_format=formats[2], gpu_gbuffer=True, gpu_vpls=True)
        if linear:
            self.driver.scene.set_field_filter(L.FIELD_LINEAR)

    def step(self, i):
        self.driver.step(i)
        return images(self.driver.session)


class Batched:
    def __init__(self, objects, preset, formats, linear):
        wl = room(objects, preset)
        self.driver = BatchDriver(Context(), [(wl, 0), (wl, 4)], *formats, use_graphs=False)
        if linear:
            for s in self.driver.scenes.values():
                s.set_field_filter(L.FIELD_LINEAR)

    def step(self, i):
        self.driver.step(i)
        return [x for v in range(2) for x in images(self.driver.batch.view(v))]


F32 = (L.GBUFFER_F32, L.RADIANCE_F32, L.MOMENTS_F32)
MIXED = (L.GBUFFER_PACKED, L.RADIANCE_F16, L.MOMENTS_F16)


@pytest.mark.parametrize("kind", [Single, Batched])
@pytest.mark.parametrize("preset,formats,linear", [(0, F32, False), (2, MIXED, False), (0, F32, True)])
def test_threads_with_small_and_large_scenes(cuda, kind, preset, formats, linear):
    sizes = (320, 3)  # 67 KB and 0.8 KB of object records
    alone = []
    for n in sizes:
        p = kind(n, preset, formats, linear)
        alone.append([p.step(i) for i in range(FRAMES)])
    threads = [ThreadPoolExecutor(1) for _ in sizes]
    programs = [t.submit(kind, n, preset, formats, linear).result() for t, n in zip(threads, sizes)]
    for i in range(FRAMES):
        for k, t in enumerate(threads):
            got = t.submit(programs[k].step, i).result()
            for a, b in zip(got, alone[k][i]):
                assert np.array_equal(a, b), (i, k)
    for t in threads:
        t.shutdown()
