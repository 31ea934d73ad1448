// capi_internal.h — the library's context, scene and session objects and
// the helpers the C-ABI translation units share (capi.cu, batch.cu).
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "dev_sdf.cuh"
#include "kernels.h"

struct irt_context {
    int device = 0;
    uint64_t budget = 0;
    std::atomic<uint64_t> in_use{0};
    mutable std::mutex mu;
    std::string last_error;
    void set_error(const std::string& e) {
        std::lock_guard<std::mutex> g(mu);
        last_error = e;
    }
};

struct irt_scene {
    irt_context* ctx = nullptr;
    uint32_t mesh_count = 0;
    irt_mesh* meshes = nullptr;
    cudaArray_t atlas_array = nullptr;
    cudaTextureObject_t atlas = 0;
    // The same atlas through a linear sampler at normalised coordinates, for
    // the reference's filtered sample_field (IRT_FIELD_LINEAR).
    cudaTextureObject_t atlas_linear = 0;
    int field_linear = 0;            // in use since the last irt_scene_update
    int field_linear_requested = 0;  // irt_scene_set_field_filter, applied by the next update
    int sdf_f16 = 0;
    // Corner cells: per field mesh, the 8 corner texels of each of its
    // (res-1)^3 cells in one record (f32: 32 B, f16: 16 B); a mesh's first
    // cell index is in hi[3] of its rows (host_meshes and the device copy).
    void* sdf_cells = nullptr;
    std::vector<irt_mesh> host_meshes;
    // per-frame data: one device block, holding every buffer below up to `cells`
    char* block = nullptr;
    uint64_t block_bytes = 0;
    irt_object* objects = nullptr;
    irt_node* nodes = nullptr;
    irt_light* lights = nullptr;
    irt_light* lights_prep = nullptr;  // spot direction normalised, cos(angle / 2)
    uint32_t object_cap = 0, light_cap = 0;
    // compact march scene (object records with their mesh and leaf box folded in)
    float4* march_scene = nullptr;
    // Pinned staging of the per-frame uploads, two slots used in turn, so an
    // update neither waits for the device nor races an earlier copy.
    unsigned char* pinned = nullptr;
    cudaEvent_t pinned_free[2] = {nullptr, nullptr};
    uint32_t updates = 0;
    // leaf-order cache (rebuilt when the BVH changes)
    uint4* cells = nullptr;
    std::vector<irt_node> cached_nodes;
    std::vector<irt_object> cached_objects;
    float grid_org[3] = {0, 0, 0}, grid_inv[3] = {0, 0, 0}, grid_size[3] = {0, 0, 0};
    float grid_slack = 0;  // error of an evaluated object distance
    uint32_t object_count = 0, light_count = 0;
    uint64_t bytes = 0;
};

// The field sampler the kernels use for a scene (point-sampled trilinear or
// the hardware-linear fetch).
inline irtd::FieldFilter scene_field_filter(const irt_scene* sc) {
    irtd::FieldFilter f{};
    f.linear = sc->field_linear ? sc->atlas_linear : 0;
    f.bound_slack = sc->field_linear ? 1.f / 32.f : sc->sdf_f16 ? 1.f / 1024.f : 0.f;
    return f;
}

struct irt_session {
    irt_context* ctx = nullptr;
    irt_session_desc desc{};
    uint32_t W = 0, H = 0;
    size_t P = 0;
    size_t rad_bytes = 0, normal_bytes = 0, mom_bytes = 0;
    char* slab = nullptr;  // the session's device memory, holding every buffer below
    irt_reservoir* dres[3] = {nullptr, nullptr, nullptr};
    irt_reservoir* ires[3] = {nullptr, nullptr, nullptr};
    irt_vpl* archive = nullptr;
    float* prev_depth = nullptr;
    void* prev_normal = nullptr;
    float4* direct = nullptr;
    void* noisy = nullptr;
    float4* moments[2] = {nullptr, nullptr};
    void* feedback[2] = {nullptr, nullptr};
    void* temporal = nullptr;
    void* scratch[2] = {nullptr, nullptr};
    void* filtered = nullptr;
    uint32_t* error = nullptr;
    uint64_t bytes = 0;
    uint32_t last_frame = 0;
    bool have_frame = false;
    bool profiling = false;
    // Profiling: a ring of kProfRing frames x 8 stage-boundary events, so a
    // long timed run can be read back afterwards without per-frame syncs.
    static constexpr int kProfRing = 128;
    static constexpr int kProfEvents = 10;
    cudaEvent_t ev[kProfRing][kProfEvents] = {};
    // ray-queue resolve buffers
    RayRecord* rays = nullptr;
    uint16_t* ray_hints = nullptr;
    float4* prep = nullptr;         // per pixel: surface normal, light of its direct ray
    uint32_t* prep_vpl = nullptr;   // per pixel: VPL of its indirect ray
    float4* ray_ends = nullptr;     // march endpoints of the pools' and the archive's VPLs, or null
    uint32_t* ray_counters = nullptr;
    float* vis = nullptr;
    float4* pending = nullptr;
    // per-pixel world positions: [0] this frame, [1] the previous frame's
    // pixels from the previous depth and previous_inv_vp
    float4* guide[2] = {nullptr, nullptr};
    float4* feat = nullptr;  // this frame's SVGF edge-stopping features, 2 float4 per pixel
    int num_sms = 0;
    // Host-input pipeline (irt_render_frame_host), created on first use:
    // a copy stream, double-buffered device G-buffers, three VPL pools plus
    // a zero pool, double-buffered device copies of the output image.
    struct HostPipe {
        bool ready = false;
        cudaStream_t copy = nullptr;      // host -> device inputs
        cudaStream_t copy_out = nullptr;  // device -> host outputs (own stream: an output copy
                                          // waits for its frame, the next inputs must not)
        void* gbuf[2] = {nullptr, nullptr};
        irt_vpl* vpls = nullptr;      // 4 pools: [0..2] ring, [3] zeros
        void* out[2] = {nullptr, nullptr};
        cudaEvent_t copied[2] = {}, rendered[2] = {}, vpl_free[3] = {}, out_ready[2] = {}, out_done[2] = {};
        cudaEvent_t march_done = nullptr;  // after the last frame's march (recorded by irt_frame_lighting)
        void* pending_out = nullptr;        // host destination of the last call's image, copied at the next call
        int pending_slot = 0;               // ... from out[pending_slot]
        uint32_t calls = 0;
        int last_vpl = -1;
        uint64_t bytes = 0;
    } pipe;
    bool ev_ready = false;
    int prof_slot = 0;
    uint32_t prof_frame[kProfRing] = {};
};

// The ray set-up of a session's frame over its scene and the caller's pools.
inline RaySetup session_ray_setup(const irt_session* s, const irt_scene* sc, const irt_vpl* cur,
                                  const irt_vpl* prev) {
    RaySetup r{};
    r.guide = s->guide[0];
    r.prep = s->prep;
    r.prep_vpl = s->prep_vpl;
    r.lights = sc->lights_prep;
    r.cur = cur;
    r.prev = prev;
    r.arch = s->archive;
    r.ends = s->ray_ends;
    r.rays = s->rays;
    r.hints = s->ray_hints;
    r.counters = s->ray_counters;
    r.vis = s->vis;
    r.vpl_count = s->desc.settings.vpl_count;
    r.slots = s->desc.settings.restir_max_history + 1u;
    return r;
}

namespace {

uint32_t normal_bytes_of(int fmt) {
    return fmt == IRT_GBUFFER_F32 ? 16u : (fmt == IRT_GBUFFER_F16 ? 8u : 4u);
}

// The error is reported here; left as the thread's last error, the next launch
// that asks for its own would report it again.
irt_status cuda_fail(irt_context* ctx, cudaError_t e, const char* what) {
    cudaGetLastError();
    if (ctx) ctx->set_error(std::string(what) + ": " + cudaGetErrorString(e));
    return IRT_E_CUDA;
}

#define CK(call, what)                                   \
    do {                                                 \
        cudaError_t _e = (call);                         \
        if (_e != cudaSuccess) return cuda_fail(ctx, _e, what); \
    } while (0)

struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev) {
        if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
        if (prev != dev) cudaSetDevice(dev);
    }
    ~DeviceGuard() {
        int cur = -1;
        if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
    }
};

template <class T>
irt_status dev_alloc(irt_context* ctx, T** p, size_t bytes, uint64_t& counter) {
    if (bytes == 0) {
        *p = nullptr;
        return IRT_OK;
    }
    void* q = nullptr;
    cudaError_t e = cudaMalloc(&q, bytes);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "cudaMalloc");
    // Zeroed when this returns: a fill left on the default stream is not
    // ordered with work that a caller's non-blocking stream does next and
    // could wipe what it has written.
    cudaStream_t fill = nullptr;
    e = cudaStreamCreateWithFlags(&fill, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMemsetAsync(q, 0, bytes, fill);
    if (e == cudaSuccess) e = cudaStreamSynchronize(fill);
    if (fill) cudaStreamDestroy(fill);
    if (e != cudaSuccess) {
        cudaFree(q);
        return cuda_fail(ctx, e, "cudaMemset");
    }
    *p = static_cast<T*>(q);
    counter += bytes;
    return IRT_OK;
}

bool needs_candidates(const irt_session_desc& d) { return d.keep_candidates || !d.fused; }

}  // namespace
