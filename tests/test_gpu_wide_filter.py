"""The allocation-free filter on frames wider than 16 bits count (it takes any
shape of up to 262144 pixels), against the sums of svgf_variance and one
svgf_atrous pass (svgf.wgsl:77-110) in f64.  The surface is one plane of one
material and colour, so every tap's edge-stopping weight is 1 and the passes
are plain box and wavelet sums; few young pixels (listed blocks of a handful)
and many (whole blocks), at both ends of the frame."""
import ctypes as C

import numpy as np
import pytest
import torch

from instantradiositytest_b200 import _lib as L
from instantradiositytest_b200.runtime import stream_handle

pytestmark = pytest.mark.gpu

# f32 sums of 49 and of 25 positive terms (2.9e-6 and, under the square root,
# 0.8e-6), approximate divisions, roots and exp2 of 1-2 ulp each
TOLERANCE = 1e-5


def expected(age, second, sigma_in):
    """Filtered sigma of one a-trous pass over the variance pass, f64."""
    h, w = age.shape
    def taps(a, r):
        padded = np.pad(a, r)
        return [(dy, dx, padded[r + dy:r + dy + h, r + dx:r + dx + w])
                for dy in range(-r, r + 1) for dx in range(-r, r + 1)]
    ones = np.ones((h, w))
    box = sum(t for _, _, t in taps(second, 3)) / sum(t for _, _, t in taps(ones, 3))
    sigma = np.where(age < 4, np.sqrt(box * 4 / np.maximum(age, 1)), sigma_in)
    kernel = {0: 1.0, 1: 2 / 3, 2: 1 / 6}
    k = lambda dy, dx: kernel[abs(dy)] * kernel[abs(dx)]
    total = sum(k(dy, dx) * t for dy, dx, t in taps(ones, 2))
    return np.sqrt(sum((k(dy, dx) * t) ** 2 for dy, dx, t in taps(sigma, 2))) / total


@pytest.mark.parametrize("width,height", [(65537, 2), (70001, 3), (200000, 1)])
@pytest.mark.parametrize("young", [0.02, 0.6])
@pytest.mark.parametrize("mfmt", [L.MOMENTS_F32, L.MOMENTS_F16])
def test_wide_frames(cuda, width, height, young, mfmt):
    rng = np.random.default_rng(width + int(young * 100))
    f = L.Frame()
    f.size[0], f.size[1] = width, height
    for m in (f.vp, f.inv_vp, f.previous_vp, f.previous_inv_vp):
        for k in range(4):
            m.m[5 * k] = 1.0
    f.camera[2] = -3.0
    age = np.where(rng.random((height, width)) < young, rng.integers(1, 4, (height, width)), 10).astype(np.float64)
    deviation = rng.integers(32, 129, (height, width)) / 64.0  # exact as a half, and its square in f32
    sigma_in = rng.uniform(0.5, 1.0, (height, width)).astype(np.float32)

    def device(a, dtype=np.float32):
        return torch.from_numpy(np.ascontiguousarray(a, dtype)).cuda()

    shape = (height, width, 1)
    depth = device(np.full((height, width), 0.25))
    normal = device(np.broadcast_to([0, 0, 1, 1], (height, width, 4)))
    color = device(np.broadcast_to([.5, .5, .5, 1], (height, width, 4)))
    params = device(np.broadcast_to([1, 0], (height, width, 2)))
    motion = device(np.zeros((height, width, 2)))
    radiance = device(np.concatenate([np.full(shape, .25), np.full(shape, .5), np.full(shape, .125),
                                      sigma_in.reshape(shape)], -1))
    if mfmt == L.MOMENTS_F32:
        moments = device(np.stack([0 * age, deviation ** 2, age, 0 * age], -1))
    else:
        words = np.zeros((height, width, 2), np.uint32)
        words[..., 0] = deviation.astype(np.float16).view(np.uint16).astype(np.uint32) << 16  # mean 0
        words[..., 1] = age.astype(np.float32).view(np.uint32)
        moments = torch.from_numpy(words.view(np.int32)).cuda()
    out = torch.full((height, width, 4), -1.0, device="cuda")
    g = L.GBuffer(L.GBUFFER_F32, depth.data_ptr(), normal.data_ptr(), color.data_ptr(), params.data_ptr(),
                  motion.data_ptr())
    err = C.create_string_buffer(256)
    status = L.lib.irt_svgf_spatial_noalloc(C.byref(f), C.byref(g), L.RADIANCE_F32, mfmt, 1, radiance.data_ptr(),
                                            moments.data_ptr(), out.data_ptr(), None, stream_handle(), err, 256)
    assert status == L.IRT_OK, err.value
    torch.cuda.synchronize()
    got = out.cpu().numpy().astype(np.float64)
    want = expected(age, deviation ** 2, sigma_in.astype(np.float64))
    assert np.all(np.abs(got[..., :3] - [.25, .5, .125]) <= TOLERANCE * .5)
    assert np.all(np.abs(got[..., 3] - want) <= TOLERANCE * want)
