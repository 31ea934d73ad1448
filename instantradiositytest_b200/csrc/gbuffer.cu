// gbuffer.cu — CUDA G-buffer producer: one primary ray per pixel centre
// against the workload's primitives (analytic boxes and spheres, or the
// triangle hierarchies of a loaded scene with back faces culled), standing in
// for the gbuffer.wgsl raster; same outputs as irt_workload_gbuffer_cpu, in f32.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <vector>

#include "dev_prims.cuh"
#include "kernels.h"
#include "workload.h"

namespace {

using irt::GPrim;

__device__ __forceinline__ void xf(const float* m, float x, float y, float z, float w, float o[4]) {
#pragma unroll
    for (int r = 0; r < 4; r++) o[r] = m[r] * x + m[4 + r] * y + m[8 + r] * z + m[12 + r] * w;
}

__device__ __forceinline__ uint16_t hbits(float v) { return __half_as_ushort(__float2half_rn(v)); }

__device__ __forceinline__ uint32_t oct_snorm16(float x, float y, float z) {
    float s = fabsf(x) + fabsf(y) + fabsf(z);
    float u = x / s, v = y / s;
    if (z < 0.f) {
        float ou = (1.f - fabsf(v)) * (u >= 0.f ? 1.f : -1.f);
        float ov = (1.f - fabsf(u)) * (v >= 0.f ? 1.f : -1.f);
        u = ou;
        v = ov;
    }
    int qu = __float2int_rn(fminf(fmaxf(u, -1.f), 1.f) * 32767.f);
    int qv = __float2int_rn(fminf(fmaxf(v, -1.f), 1.f) * 32767.f);
    return ((uint32_t)(uint16_t)(int16_t)qu) | ((uint32_t)(uint16_t)(int16_t)qv << 16);
}

// Ray of the image point (u, v): d spans near to far plane, t in [0, 1).  w:
// the homogeneous coordinates of the two points.
__device__ __forceinline__ void primary_ray(const irt_frame& f, float u, float v, float o[3], float d[3], float w[2]) {
    float nx = u * 2.f - 1.f, ny = 1.f - v * 2.f;
    float pn[4], pf[4];
    xf(f.inv_vp.m, nx, ny, 0.f, 1.f, pn);
    xf(f.inv_vp.m, nx, ny, 1.f, 1.f, pf);
#pragma unroll
    for (int a = 0; a < 3; a++) {
        o[a] = pn[a] / pn[3];
        d[a] = pf[a] / pf[3] - o[a];
    }
    w[0] = pn[3];
    w[1] = pf[3];
}

// Primitives a block of pixels may see, in ascending order: those whose
// bounding sphere is not wholly beyond one of the four planes through the rays
// of neighbouring block corners.  Every pixel of the block tests the same few
// primitives instead of all: 1280x720, 23 objects 97 -> 57 us, 2560x1600, 50
// objects 816 -> 303.
//
// The planes hold for every inv_vp, parallel projections among them: a plane
// goes through both corners' near and far points (parallel image lines stay
// coplanar), and its outer side follows from the sign of inv_vp's determinant
// (`orientation`, from the host), which a block too narrow for f32 cannot get
// wrong.  What f32 makes of the corners, and of the pixels' own rays, goes into
// each plane's slack.  A block whose homogeneous w changes its sign is not the
// hull of its corners and keeps all primitives, as does anything not finite.
constexpr uint32_t kMaxListed = 2048;
// What the lists of a frame need of its inv_vp besides the rays.
struct ListFrame {
    float orientation;     // sign of the determinant; 0: no planes
    float near_sum, far_sum;  // length of the sums of |products| behind a near and a far point
    float w_sum;           // the same of w, or 0 where every pixel has the same bits of w
};
struct BlockPrims {
    float corner_o[4][3], corner_d[4][3];
    float plane[4][3];  // unit normal, outward; 0 = no plane
    float slack[4];     // of a distance from the plane, per distance from its corner
    uint32_t count;
    uint16_t index[kMaxListed];
};
__device__ __forceinline__ bool beyond(const BlockPrims& s, const GPrim& p) {
    // bounding sphere in world space: the model's largest stretch is at most
    // sqrt of the largest row sum of |A^T A|
    float m[3], half;
    if (p.kind == irt::kPrimSphere) {
        m[0] = m[1] = m[2] = 0.f;
        half = p.lo[0];
    } else {
        float h2 = 0.f;
        for (int a = 0; a < 3; a++) {
            m[a] = .5f * (p.lo[a] + p.hi[a]);
            const float h = .5f * (p.hi[a] - p.lo[a]);
            h2 += h * h;
        }
        half = sqrtf(h2);
    }
    float c[4];
    xf(p.model, m[0], m[1], m[2], 1.f, c);
    float stretch = 0.f;
    for (int a = 0; a < 3; a++) {
        float row = 0.f;
        for (int b = 0; b < 3; b++) {
            float dot = 0.f;
            for (int k = 0; k < 3; k++) dot += p.model[4 * a + k] * p.model[4 * b + k];
            row += fabsf(dot);
        }
        stretch = fmaxf(stretch, row);
    }
    const float r = 1.01f * half * sqrtf(stretch);
    for (int k = 0; k < 4; k++) {
        const float *n = s.plane[k], *o = s.corner_o[k];
        const float w[3] = {c[0] - o[0], c[1] - o[1], c[2] - o[2]};
        const float away = sqrtf(w[0] * w[0] + w[1] * w[1] + w[2] * w[2]) + r;
        if (n[0] * w[0] + n[1] * w[1] + n[2] * w[2] > r + s.slack[k] * away + 1e-3f) return true;
    }
    return false;
}
// The plane through corner t of the block's pixels and the next in their
// cycle; by lanes 0-3.
__device__ __forceinline__ void block_plane(const irt_frame& f, const ListFrame& lf, uint32_t t, BlockPrims& s) {
    const unsigned lanes = 0xfu;
    const float W = (float)f.size[0], H = (float)f.size[1];
    const float x = (float)((blockIdx.x + (t == 1u || t == 2u ? 1u : 0u)) * blockDim.x);
    const float y = (float)((blockIdx.y + (t >= 2u ? 1u : 0u)) * blockDim.y);
    float o[3], d[3], w[2], v[3], norm[2];
    primary_ray(f, fminf(x, W) / W, fminf(y, H) / H, o, d, w);
    // |a coordinate's error| <= 4 roundings of its sum, the same of w, one
    // division: 2^-22 of them; as much again for the pixels' own rays.
    norm[0] = fabsf(o[0]) + fabsf(o[1]) + fabsf(o[2]);
    norm[1] = fabsf(o[0] + d[0]) + fabsf(o[1] + d[1]) + fabsf(o[2] + d[2]);
    const float e = 0x1p-21f * (__fdividef(lf.near_sum + norm[0] * lf.w_sum, fabsf(w[0])) + norm[0] +
                                __fdividef(lf.far_sum + norm[1] * lf.w_sum, fabsf(w[1])) + norm[1]);
    const bool hull = __all_sync(lanes, w[0] > 0.f && w[1] > 0.f) || __all_sync(lanes, w[0] < 0.f && w[1] < 0.f);
    const int next = (int)((t + 1u) & 3u);
#pragma unroll
    for (int i = 0; i < 3; i++) {
        s.corner_o[t][i] = o[i];
        s.corner_d[t][i] = d[i];
        v[i] = __shfl_sync(lanes, o[i] + d[i], next) - o[i];
    }
    const float n[3] = {d[1] * v[2] - d[2] * v[1], d[2] * v[0] - d[0] * v[2], d[0] * v[1] - d[1] * v[0]};
    const float inv = rsqrtf(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
    const float ld = fabsf(d[0]) + fabsf(d[1]) + fabsf(d[2]), lv = fabsf(v[0]) + fabsf(v[1]) + fabsf(v[2]);
    const float error = fmaxf(e, __shfl_sync(lanes, e, next)) * (ld + lv) + 0x1p-21f * ld * lv;
#pragma unroll
    for (int i = 0; i < 3; i++) s.plane[t][i] = hull ? n[i] * (lf.orientation * inv) : 0.f;
    s.slack[t] = .002f + error * inv;
}
__device__ __forceinline__ void list_block_prims(const irt_frame& f, const ListFrame& lf, const irt::PrimTable& T,
                                                 BlockPrims& s) {
    const uint32_t t = threadIdx.y * blockDim.x + threadIdx.x;
    if (t < 32u) {
        if (t < 4u) block_plane(f, lf, t, s);
        __syncwarp();
        uint32_t count = 0;
        for (uint32_t first = 0; first < T.n; first += 32u) {
            const bool keep = first + t < T.n && !beyond(s, T.prims[first + t]);
            const unsigned kept = __ballot_sync(0xffffffffu, keep);
            if (keep) s.index[count + __popc(kept & ((1u << t) - 1u))] = (uint16_t)(first + t);
            count += (uint32_t)__popc(kept);
        }
        if (t == 0u) s.count = count;
    }
    __syncthreads();
}

__global__ void gbuffer_kernel(const __grid_constant__ irt_frame f, const __grid_constant__ ListFrame lf, const irt::PrimTable T,
                               int fmt, float* depth, void* normal, void* color, void* params, void* motion) {
    __shared__ BlockPrims listed;
    const bool list = T.n <= kMaxListed;
    if (list) list_block_prims(f, lf, T, listed);
    uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t y = blockIdx.y * blockDim.y + threadIdx.y;
    uint32_t W = f.size[0], H = f.size[1];
    if (x >= W || y >= H) return;
    size_t i = (size_t)y * W + x;
    float u = ((float)x + .5f) / (float)W, v = ((float)y + .5f) / (float)H;
    float o[3], d[3], hw[2];
    primary_ray(f, u, v, o, d, hw);
    float best;
    float nl_best[3] = {0, 0, 0};
    int hit = irtd::cast_prims(T, list ? listed.count : T.n, [&](uint32_t j) { return list ? (uint32_t)listed.index[j] : j; },
                               o, d, 0.f, 1.f, true, best, nl_best);
    float dep = 1.f, nrm[3] = {0, 0, 0}, col[3] = {0, 0, 0}, par[2] = {0, 0}, mot[2] = {0, 0};
    if (hit >= 0) {
        const GPrim& p = T.prims[hit];
        float w[4];
        xf(p.model, nl_best[0], nl_best[1], nl_best[2], 0.f, w);
        float inv = 1.f / sqrtf(w[0] * w[0] + w[1] * w[1] + w[2] * w[2]);
        nrm[0] = w[0] * inv;
        nrm[1] = w[1] * inv;
        nrm[2] = w[2] * inv;
        float P[3] = {o[0] + d[0] * best, o[1] + d[1] * best, o[2] + d[2] * best};
        float c[4], pc[4];
        xf(f.vp.m, P[0], P[1], P[2], 1.f, c);
        xf(f.previous_vp.m, P[0], P[1], P[2], 1.f, pc);
        dep = fminf(c[2] / c[3], 0.99999994f);
        col[0] = p.color[0];
        col[1] = p.color[1];
        col[2] = p.color[2];
        par[0] = p.params[0];
        par[1] = p.params[1];
        mot[0] = (c[0] / c[3] - pc[0] / pc[3]) * .5f;
        mot[1] = (c[1] / c[3] - pc[1] / pc[3]) * -.5f;
    }
    float alpha = hit >= 0 ? 1.f : 0.f;
    depth[i] = dep;
    if (fmt == IRT_GBUFFER_F32) {
        ((float4*)normal)[i] = make_float4(nrm[0], nrm[1], nrm[2], alpha);
        ((float4*)color)[i] = make_float4(col[0], col[1], col[2], alpha);
        ((float2*)params)[i] = make_float2(par[0], par[1]);
        ((float2*)motion)[i] = make_float2(mot[0], mot[1]);
    } else if (fmt == IRT_GBUFFER_F16) {
        ((uint2*)normal)[i] = make_uint2(hbits(nrm[0]) | ((uint32_t)hbits(nrm[1]) << 16), hbits(nrm[2]) | ((uint32_t)hbits(alpha) << 16));
        ((uint2*)color)[i] = make_uint2(hbits(col[0]) | ((uint32_t)hbits(col[1]) << 16), hbits(col[2]) | ((uint32_t)hbits(alpha) << 16));
        ((uint32_t*)params)[i] = hbits(par[0]) | ((uint32_t)hbits(par[1]) << 16);
        ((uint32_t*)motion)[i] = hbits(mot[0]) | ((uint32_t)hbits(mot[1]) << 16);
    } else {
        ((uint32_t*)normal)[i] = hit >= 0 ? oct_snorm16(nrm[0], nrm[1], nrm[2]) : 0u;
        auto q8 = [](float c) { return (uint32_t)__float2int_rn(fminf(fmaxf(c, 0.f), 1.f) * 255.f); };
        ((uint32_t*)color)[i] = q8(col[0]) | (q8(col[1]) << 8) | (q8(col[2]) << 16) | (q8(alpha) << 24);
        ((uint32_t*)params)[i] = hbits(par[0]) | ((uint32_t)hbits(par[1]) << 16);
        ((uint32_t*)motion)[i] = hbits(mot[0]) | ((uint32_t)hbits(mot[1]) << 16);
    }
}

ListFrame list_frame(const float* m) {
    ListFrame lf{};
    auto minor = [&](int r, int a, int b) {  // rows r and r + 1, columns a and b
        return (double)m[4 * a + r] * m[4 * b + r + 1] - (double)m[4 * b + r] * m[4 * a + r + 1];
    };
    const double det = minor(0, 0, 1) * minor(2, 2, 3) - minor(0, 0, 2) * minor(2, 1, 3) + minor(0, 0, 3) * minor(2, 1, 2) +
                       minor(0, 1, 2) * minor(2, 0, 3) - minor(0, 1, 3) * minor(2, 0, 2) + minor(0, 2, 3) * minor(2, 0, 1);
    lf.orientation = det > 0 ? 1.f : det < 0 ? -1.f : 0.f;
    double near2 = 0, far2 = 0;
    for (int a = 0; a < 3; a++) {
        const double near_a = std::fabs(m[a]) + std::fabs(m[4 + a]) + std::fabs(m[12 + a]);
        near2 += near_a * near_a;
        far2 += (near_a + std::fabs(m[8 + a])) * (near_a + std::fabs(m[8 + a]));
    }
    lf.near_sum = (float)std::sqrt(near2);
    lf.far_sum = (float)std::sqrt(far2);
    // x and y too small to reach the sum's last bit leave w the same everywhere
    const double xy = std::fabs(m[3]) + std::fabs(m[7]), z = std::fabs(m[11]), one = std::fabs(m[15]);
    const bool same = xy <= 0x1p-26 * one && (z == 0 || xy <= 0x1p-26 * z);
    lf.w_sum = same ? 0.f : (float)(xy + z + one);
    return lf;
}

}  // namespace

// Flattened primitive table of a workload on the current device (static
// scenes: built once and kept with the workload), with the triangle
// hierarchies of loaded meshes concatenated into shared node and triangle
// tables.
// Frees a workload's device primitive tables (Workload::release_device).
static void release_prims(irt::Workload& w) {
    int prev = -1;
    cudaGetDevice(&prev);
    const bool other = w.dev_prims_device >= 0 && prev != w.dev_prims_device;
    if (other) cudaSetDevice(w.dev_prims_device);
    for (void* p : {w.dev_prims, w.dev_nodes, w.dev_tris})
        if (p) cudaFree(p);
    w.dev_prims = w.dev_nodes = w.dev_tris = nullptr;
    if (other && prev >= 0) cudaSetDevice(prev);
}

cudaError_t irt_workload_prims(const irt_workload* wl_c, irt::PrimTable* out) {
    irt_workload* wl = const_cast<irt_workload*>(wl_c);
    irt::Workload& w = wl->w;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (!w.dev_prims || w.dev_prims_device != dev) {
        std::vector<GPrim> prims;
        std::vector<irt::TriNode> nodes;
        std::vector<irt::TriRec> tris;
        std::vector<uint32_t> node_base(w.mesh_desc.size(), 0), tri_base(w.mesh_desc.size(), 0);
        for (size_t m = 0; m < w.mesh_desc.size(); m++) {
            const irt::MeshDesc& md = w.mesh_desc[m];
            if (!md.triangles) continue;
            node_base[m] = (uint32_t)nodes.size();
            tri_base[m] = (uint32_t)tris.size();
            nodes.insert(nodes.end(), md.bvh.nodes.begin(), md.bvh.nodes.end());
            tris.insert(tris.end(), md.bvh.tris.begin(), md.bvh.tris.end());
        }
        for (uint32_t oi = 0; oi < w.objs.size(); oi++) {
            const irt::Obj& ob = w.objs[oi];
            irt_mat4 model = irt::to_f32(ob.model), inv = irt::to_f32(ob.inv_model);
            const irt_material& m = w.materials[ob.material];
            const irt::MeshDesc& md = w.mesh_desc[ob.mesh];
            GPrim g{};
            for (int k = 0; k < 16; k++) {
                g.inv_model[k] = inv.m[k];
                g.model[k] = model.m[k];
            }
            for (int k = 0; k < 3; k++) g.color[k] = m.color[k];
            g.params[0] = fminf(fmaxf(m.params[0], .045f), 1.f);
            g.params[1] = fminf(fmaxf(m.params[1], 0.f), 1.f);
            g.object = oi;
            if (md.triangles) {
                if (md.bvh.nodes.empty()) continue;
                g.kind = irt::kPrimTriangles;
                for (int a = 0; a < 3; a++) {
                    g.lo[a] = md.bvh.nodes[0].lo[a];
                    g.hi[a] = md.bvh.nodes[0].hi[a];
                }
                g.node_base = node_base[ob.mesh];
                g.tri_base = tri_base[ob.mesh];
                prims.push_back(g);
                continue;
            }
            for (const irt::Part& part : md.parts) {
                for (int a = 0; a < 3; a++) {
                    g.lo[a] = part.sphere ? 0.f : (float)part.lo[a];
                    g.hi[a] = part.sphere ? 0.f : (float)part.hi[a];
                }
                if (part.sphere) g.lo[0] = (float)part.radius;
                g.kind = part.sphere ? irt::kPrimSphere : irt::kPrimBox;
                prims.push_back(g);
            }
        }
        for (void** p : {&w.dev_prims, &w.dev_nodes, &w.dev_tris}) {
            if (*p) cudaFree(*p);
            *p = nullptr;
        }
        w.dev_prims_count = 0;
        w.release_device = &release_prims;
        auto upload = [](void** dst, const void* src, size_t bytes) {
            if (bytes == 0) return cudaSuccess;
            cudaError_t r = cudaMalloc(dst, bytes);
            if (r != cudaSuccess) return r;
            r = cudaMemcpy(*dst, src, bytes, cudaMemcpyHostToDevice);
            // a caller's non-blocking stream does not wait for the default one
            return r == cudaSuccess ? cudaStreamSynchronize(nullptr) : r;
        };
        e = upload(&w.dev_prims, prims.data(), prims.size() * sizeof(GPrim));
        if (e == cudaSuccess) e = upload(&w.dev_nodes, nodes.data(), nodes.size() * sizeof(irt::TriNode));
        if (e == cudaSuccess) e = upload(&w.dev_tris, tris.data(), tris.size() * sizeof(irt::TriRec));
        if (e != cudaSuccess) return e;
        w.dev_prims_device = dev;
        w.dev_prims_count = (uint32_t)prims.size();
    }
    out->prims = static_cast<const GPrim*>(w.dev_prims);
    out->n = w.dev_prims_count;
    out->nodes = static_cast<const irt::TriNode*>(w.dev_nodes);
    out->tris = static_cast<const irt::TriRec*>(w.dev_tris);
    return cudaSuccess;
}

extern "C" irt_status irt_gbuffer_render(irt_context* ctx, const irt_workload* wl, const irt_frame* f,
                                         const irt_object* objects, int32_t format, float* depth, void* normal,
                                         void* color, void* params, void* motion, void* stream) {
    (void)objects;
    if (!ctx || !wl || !f || !depth || !normal || !color || !params || !motion) return IRT_E_INVALID;
    if (format < IRT_GBUFFER_F32 || format > IRT_GBUFFER_PACKED) return IRT_E_INVALID;
    irt::PrimTable T{};
    if (irt_workload_prims(wl, &T) != cudaSuccess) return IRT_E_CUDA;
    dim3 block(32, 8);
    dim3 grid((f->size[0] + 31) / 32, (f->size[1] + 7) / 8);
    gbuffer_kernel<<<grid, block, 0, static_cast<cudaStream_t>(stream)>>>(
        *f, list_frame(f->inv_vp.m), T, format, depth, normal, color, params, motion);
    return cudaGetLastError() == cudaSuccess ? IRT_OK : IRT_E_CUDA;
}
