"""A batch renders each view with its own frame's march parameters (steps, hit
epsilon, soft-shadow k): views of one scene that differ in them, and frames
that change them after the batch's graphs were captured, equal the view's
render alone."""
import numpy as np
import pytest
import torch

from instantradiositytest_b200 import _lib as L
from instantradiositytest_b200.batching import BatchDriver
from instantradiositytest_b200.runtime import Context

from test_gpu_batch import BUFS, render_alone, workload

pytestmark = pytest.mark.gpu


def own_parameters(v, i):
    """Two of three views of a scene differ."""
    return [(0, 1.0), (1, 3.0), (2, 0.25)][v % 3] if v % 3 else None


def later_parameters(v, i):
    """From frame 6 on (graphs replay from frame 4) every view's differ from before."""
    return (2, 0.2) if i >= 6 else None


@pytest.mark.parametrize("change", [own_parameters, later_parameters])
def test_views_march_with_their_own_parameters(cuda, change):
    a, b = workload(71, 9, 160, 100), workload(72, 6, 96, 64)
    views = [(a, 0), (a, 5), (a, 9), (b, 1), (b, 6)]
    ctx = Context()
    drv = BatchDriver(ctx, views, use_graphs=True)
    per_view = [[] for _ in views]
    replayed = []
    for i in range(10):
        data = drv.inputs(i)
        for v, (f, *_) in enumerate(data):
            scaled = change(v, i)
            if scaled:
                f.sdf[scaled[0]] *= scaled[1]
        frames = drv.step(i, data)
        for v, (f, (_, obj, nodes, lights)) in enumerate(zip(frames, data)):
            per_view[v].append((L.Frame.from_buffer_copy(f), obj, nodes, lights))
        torch.cuda.synchronize()
        replayed.append(drv.batch.pass_ms()["graph"])
    assert replayed[5] == 1.0 and replayed[9] == 1.0
    plain = {}
    for v, (wl, _) in enumerate(views):
        s = drv.batch.view(v)
        ref = render_alone(ctx, wl, per_view[v], L.GBUFFER_F32, L.RADIANCE_F32, L.MOMENTS_F32)
        for w in BUFS:
            assert np.array_equal(s.buffer(w, torch.uint8).cpu().numpy(), ref[w]), (v, w)
        plain[v] = ref[L.BUF_NOISY]
    # the changed parameters show in the images: the test compares something
    v = 1
    for f, *_ in per_view[v]:
        f.sdf[:] = drv.inputs(0)[v][0].sdf[:]
    ref = render_alone(ctx, views[v][0], per_view[v], L.GBUFFER_F32, L.RADIANCE_F32, L.MOMENTS_F32)
    assert not np.array_equal(plain[v], ref[L.BUF_NOISY])
    drv.close()
    ctx.close()
