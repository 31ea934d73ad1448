"""A batch over more scenes than one march launch takes (16): one launch for
the first 16, another for the rest, and every view equal to its render alone,
with direct launches and graph replays."""
import numpy as np
import pytest
import torch

from instantradiositytest_b200 import _lib as L
from instantradiositytest_b200.batching import BatchDriver
from instantradiositytest_b200.runtime import Context

from test_gpu_batch import BUFS, render_alone, workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scenes", [16, 17])
def test_batch_of_many_scenes_equals_alone(cuda, scenes):
    wls = [workload(60 + k, 3 + k % 3, 96 - 8 * (k % 2), 64) for k in range(scenes)]
    views = [(wl, k) for k, wl in enumerate(wls)] + [(wls[-1], 5)]
    ctx = Context()
    drv = BatchDriver(ctx, views, use_graphs=True)
    per_view = [[] for _ in views]
    for i in range(6):
        data = drv.inputs(i)
        frames = drv.step(i, data)
        for v, (f, (_, obj, nodes, lights)) in enumerate(zip(frames, data)):
            per_view[v].append((L.Frame.from_buffer_copy(f), obj, nodes, lights))
    torch.cuda.synchronize()
    assert drv.batch.pass_ms()["graph"] == 1.0
    for v, (wl, _) in enumerate(views):
        s = drv.batch.view(v)
        ref = render_alone(ctx, wl, per_view[v], L.GBUFFER_F32, L.RADIANCE_F32, L.MOMENTS_F32)
        for w in BUFS:
            assert np.array_equal(s.buffer(w, torch.uint8).cpu().numpy(), ref[w]), (v, w)
    drv.close()
    ctx.close()
