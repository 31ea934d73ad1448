"""normalize() of the device code (three quotients from one reciprocal,
dev_common.cuh) against CUDA's own division, bit for bit: a harness compiled
with the lighting kernels' flags divides by the same length both ways.  Over
all lengths whose squares f32 holds, and for zero, infinite and not-a-number
components.  Components below
2^-100 are left out: there the correction's residual leaves the normal range and
a last bit may differ."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HARNESS = r"""
#include <cuda_runtime.h>
#include "dev_common.cuh"
using namespace irtd;
__global__ void both(const float* v, float* ours, float* cuda, unsigned n) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const V3 a{v[3 * i], v[3 * i + 1], v[3 * i + 2]};
    const V3 q = normalize(a);
    const float s = sqrtf(dot(a, a));
    ours[3 * i] = q.x, ours[3 * i + 1] = q.y, ours[3 * i + 2] = q.z;
    cuda[3 * i] = __fdiv_rn(a.x, s), cuda[3 * i + 1] = __fdiv_rn(a.y, s), cuda[3 * i + 2] = __fdiv_rn(a.z, s);
}
extern "C" int run(const float* v, float* ours, float* cuda, unsigned n) {
    both<<<(n + 255) / 256, 256>>>(v, ours, cuda, n);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("division")
    src, lib = d / "division.cu", d / "libdivision.so"
    src.write_text(HARNESS)
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    pkg = os.path.join(ROOT, "instantradiositytest_b200", "csrc")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "-I", pkg, "-I", os.path.join(ROOT, "include"), str(src), "-o", str(lib)], check=True)
    return C.CDLL(str(lib))


def quotients(harness, v):
    d = torch.from_numpy(np.ascontiguousarray(v, np.float32)).cuda()
    ours, cuda = torch.empty_like(d), torch.empty_like(d)
    assert harness.run(C.c_void_p(d.data_ptr()), C.c_void_p(ours.data_ptr()), C.c_void_p(cuda.data_ptr()),
                       len(v)) == 0
    return ours.cpu().numpy(), cuda.cpu().numpy()


@pytest.mark.parametrize("seed", range(4))
def test_normalize_equals_division(cuda, harness, seed):
    rng = np.random.default_rng(seed)
    n = 1 << 22
    length = np.exp2(rng.uniform(-45, 49, n))
    v = rng.normal(size=(n, 3))
    v *= (length / np.linalg.norm(v, axis=1))[:, None]
    v[: n // 4, 0] *= np.exp2(-rng.uniform(0, 100, n // 4))
    v[n // 4:n // 2, 1:] = 0.0
    v[n // 2:n // 2 + 4096] = np.sign(v[n // 2:n // 2 + 4096])
    ours, cuda_ = quotients(harness, v)
    tiny = (v != 0) & (np.abs(v) < np.exp2(-100))
    assert tiny.mean() < 0.05
    same = ours.view(np.uint32) == cuda_.view(np.uint32)
    assert np.all(same | tiny), (v[(~(same | tiny)).any(1)][:4], ours[(~(same | tiny)).any(1)][:4])


def test_extreme_lengths(cuda, harness):
    edge = [0.0, -0.0, np.inf, -np.inf, np.nan, 1e-30, 1e-22, 9.9e-16, 1e-15, 1.1e-15, 1e-3, 1.0, 9.9e14, 1e15, 1.1e15,
            1e18, 1.8e19, 3e19, 3e38]
    v = np.array([(a, b, c) for a in edge for b in edge for c in edge], np.float32)
    ours, cuda_ = quotients(harness, v)
    # the same infinities, zeros and NaNs, and the same quotients
    assert np.array_equal(np.isnan(ours), np.isnan(cuda_))
    ok = np.isfinite(cuda_)
    assert np.array_equal(ours[~ok & ~np.isnan(cuda_)], cuda_[~ok & ~np.isnan(cuda_)])
    normal = ok & (np.abs(cuda_) >= 2.0 ** -100) & (np.abs(v) >= 2.0 ** -100)
    assert np.array_equal(ours[normal], cuda_[normal])
