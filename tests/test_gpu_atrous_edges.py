"""The SVGF spatial passes where their branches meet.  A-trous: taps reach 2 x
step pixels (steps 1 to 16), so a frame narrower than 4 x step has no interior
pixel at that step, and blocks of 256 pixels of a row end in ragged ones.
Variance: every pixel of a block young (the first frames), and, under a camera
that moves on, blocks with a few young pixels or none.  Lockstep with the
oracle, every storage, the repository's radiance bar."""
import pytest

from instantradiositytest_b200 import _lib as L
from instantradiositytest_b200.workload import Workload

from gpu_harness import RADIANCE_BAR, SELECT_BAR, Lockstep

pytestmark = pytest.mark.gpu

STORAGE = {"f32": (L.GBUFFER_F32, L.RADIANCE_F32, L.MOMENTS_F32), "f16": (L.GBUFFER_F16, L.RADIANCE_F16, L.MOMENTS_F32),
           "mixed": (L.GBUFFER_PACKED, L.RADIANCE_F16, L.MOMENTS_F16)}


@pytest.mark.parametrize("storage", list(STORAGE))
@pytest.mark.parametrize("size,iterations", [((5, 3), 1), ((33, 9), 5), ((66, 67), 5), ((257, 33), 4), ((300, 65), 5)])
def test_atrous_at_frame_edges(cuda, storage, size, iterations):
    wl = Workload(0, width=size[0], height=size[1], n_lights=2)
    wl.settings.svgf_iterations = iterations
    g, r, m = STORAGE[storage]
    lock = Lockstep(wl, gbuffer_format=g, radiance_format=r, moments_format=m)
    for i in range(3):
        got = lock.frame(i)
        assert got["filtered"] <= RADIANCE_BAR, (i, got)
        assert got["select_d2"] >= SELECT_BAR and got["select_i2"] >= SELECT_BAR, (i, got)
    lock.close()
    wl.close()


@pytest.mark.parametrize("storage", list(STORAGE))
def test_variance_of_few_young_pixels(cuda, storage):
    wl = Workload(0, width=97, height=61, n_boxes=6, n_spheres=4, orbit_deg_per_frame=1.5)
    g, r, m = STORAGE[storage]
    lock = Lockstep(wl, gbuffer_format=g, radiance_format=r, moments_format=m)
    for i in range(9):
        got = lock.frame(i)
        assert got["filtered"] <= RADIANCE_BAR, (i, got)
    age = lock.drv.session.moments_host()[..., 2]
    young = (age < 4).mean()
    assert 0.0 < young < 0.5, young  # disoccluded edges beside a settled image
    lock.close()
    wl.close()
