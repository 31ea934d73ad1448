// kernels.h — host-side launch descriptors of the lighting and SVGF kernels.
#pragma once
#include <cuda_runtime.h>

#include "../../include/irt.h"
#include "workload.h"

namespace irtd {
// The reference's filtered variant of sample_field (src/renderer.rs:277-286,
// chosen there whenever the adapter can filter R32Float textures): one
// hardware-linear fetch of the atlas at the point (origin + q + .5) / dims in
// normalised coordinates — texel coordinate origin + q + .5 — clamp-to-edge,
// instead of 8 texel loads and f32 weights.  linear == 0 selects the
// point-sampled trilinear of common.wgsl:31-38.
struct FieldFilter {
    cudaTextureObject_t linear;  // the atlas: texel coordinates, linear filter, clamp
    // Voxels by which a sampled distance may miss the trilinear value of the
    // exact field, for the leaf-order cache's bounds: three axes of 8-bit weights
    // for the filtered sampler; an f16 texel's 2^-10 of its value, which exceeds
    // the distance by half a voxel and within a cell by up to one (the part that
    // grows with the distance is in the cache's slope); 0 for f32 points.
    float bound_slack;
};
}  // namespace irtd

// Launch of a frame's kernel behind the one before it in its stream
// (programmatic dependent launch): its blocks may become resident once every
// block of that kernel has started its work, and wait_for_previous() at the
// kernel's start holds them until that kernel has completed and its writes are
// visible; after it, let_next_start() opens the same to the next one.  Every
// kernel launched so calls both, in this order, before it touches memory the
// frame writes, so a kernel's completion implies that of all before it.  What
// is saved is the launch and ramp-up between kernels.
//
// A kernel launched behind another is resident while that one still writes, so
// what that one may write is read by ordinary loads (load_written,
// dev_common.cuh): the non-coherent path, __ldg and const __restrict__, is for
// data that nobody writes during a kernel's lifetime, and its loads may be moved
// above the wait.  What kernels further back wrote is complete by then.  The
// ordinary loads cost the denoiser alone 821 -> 830 us at 1920x1080 f16 and a
// 480x300 frame 402 -> 404; larger frames take what they took.
template <class... P, class... A>
inline cudaError_t launch_behind(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = st;
    cudaLaunchAttribute a{};
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &a;
    c.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
    if (e != cudaSuccess) cudaGetLastError();  // returned here, not to the next launch's check
    return e;
}
#ifdef __CUDACC__
namespace irtd {
__device__ __forceinline__ void wait_for_previous() { cudaGridDependencySynchronize(); }
__device__ __forceinline__ void let_next_start() { cudaTriggerProgrammaticLaunchCompletion(); }
__device__ __forceinline__ void frame_kernel_begin() {
    wait_for_previous();
    let_next_start();
}
}  // namespace irtd
#endif

// Lighting stages: 0..7 are the reference entry points in schedule order
// (candidates_direct, candidates_indirect, temporal_direct, temporal_indirect,
// spatial_direct, spatial_indirect, resolve_direct, resolve_indirect).
constexpr int kStageReuse = 100;    // fused 0..3
constexpr int kStageShade = 101;    // fused 4..7 with the march inline (one thread per pixel)
constexpr int kStageSpatial = 102;  // fused 4..5 + resolve set-up: names each pixel's visibility rays
constexpr int kStageCombine = 103;  // resolve 6..7 from contributions x visibility

// A visibility ray of the resolve passes (sdf.wgsl:61-81) as its march
// begins, 32 bytes: a = (origin.xyz, bits(pixel * 2 + kind)) with the surface
// clearance applied, kind 0 = direct, 1 = indirect; b = (direction.xyz,
// length).  The object nearest the surface point (the march's first hint) is
// in a 16-bit array beside the records.
struct RayRecord {
    float4 a, b;
};

// What the ray set-up of a frame reads and writes (march.cu).
struct RaySetup {
    // From the spatial pass, per pixel: prep = (surface normal, bits(light id
    // of its direct ray)), prep_vpl = VPL of its indirect ray; kNoRay = none.
    // VPL v < vpl_count is entry v of the current pool, v < 2 * vpl_count
    // entry v - vpl_count of the previous one, else of the archive.
    const float4* guide;
    float4* prep;
    uint32_t* prep_vpl;
    const irt_light* lights;
    const irt_vpl* cur;
    const irt_vpl* prev;
    irt_vpl* arch;
    // March endpoints of every VPL (the same order), or null: one query per ray.
    float4* ends;
    RayRecord* rays;     // capacity 2 * W * H
    uint16_t* hints;     // capacity 2 * W * H
    uint32_t* counters;  // [0] VPL rays (queue front), [1] rays fetched by the march, [2] light rays (back)
    float* vis;          // visibility per pixel * 2 + kind
    uint32_t vpl_count, slots;
};
constexpr uint32_t kNoRay = 0xffffffffu;
// VPLs whose endpoints a session tabulates: the two pools and the archive.
inline uint64_t irt_ray_pool_entries(uint32_t vpl_count, uint32_t max_history) {
    return (uint64_t)vpl_count * (max_history + 3u);
}

struct LightingLaunch {
    const irt_frame* frame;
    irt_gbuffer gbuffer;
    const irt_object* objects;
    const irt_mesh* meshes;
    const irt_node* nodes;
    const irt_light* lights;
    cudaTextureObject_t atlas;
    int sdf_f16;
    const void* sdf_cells;  // corner cells of the field meshes (dev_sdf.cuh), or null
    irtd::FieldFilter field_filter;
    uint32_t* error;
    const irt_vpl* cur_vpls;
    const irt_vpl* prev_vpls;
    const irt_vpl* archive;
    const void* prev_normal;
    irt_reservoir* dres[3];
    irt_reservoir* ires[3];
    float4* direct_out;
    void* noisy_out;
    int radiance_f16;
    int keep_candidates;
    const float4* guide;      // world positions of this frame's pixels
    const float4* old_guide;  // ... of the previous frame's pixels
    const float4* feat;       // decoded normal/colour/params of this frame's pixels (f16, packed), or null
    // ray-queue resolve (kStageSpatial / march / kStageCombine)
    float4* prep;            // per pixel (RaySetup)
    uint32_t* prep_vpl;
    float* vis;              // visibility per pixel * 2 + kind
    float4* pending;         // per pixel: direct contribution (w = 1: x vis), indirect (w = 1: x vis)
};

struct MarchLaunch {
    const irt_frame* frame;
    const irt_object* objects;
    const irt_mesh* meshes;
    const irt_node* nodes;
    cudaTextureObject_t atlas;
    int sdf_f16;
    const void* sdf_cells;  // corner cells of the field meshes (dev_sdf.cuh), or null
    irtd::FieldFilter field_filter;
    uint32_t* error;
    const float4* march_scene;  // object records (irt_march_scene_bytes)
    // Leaf-order cache: a kGridRes^3 grid over the root box; per cell the
    // first kCellEntries objects by increasing lower bound of their distance
    // from the cell's centre, those bounds and the next one as a sentinel.
    const uint4* cells;
    float grid_org[3], grid_inv[3], grid_size[3], grid_slack;
    RaySetup setup;
    int num_sms;
    int fast;  // 1: approximate division / square root build (march_fast.cu)
};
// The frame's VPL archive slot, ray-counter reset and VPL endpoints (before
// the lighting passes); the ray set-up and the march (after them).
cudaError_t irt_launch_ray_pools(const MarchLaunch& M, cudaStream_t st);
cudaError_t irt_launch_march(const MarchLaunch& M, cudaStream_t st);
// Bytes of the compact march scene of `object_count` objects: records of 208
// bytes (dev_sdf.cuh: MObj).
uint32_t irt_march_scene_bytes(uint32_t object_count);
constexpr uint32_t kMaxMarchObjects = 1024;  // the march scene lives in shared memory
constexpr uint32_t kGridRes = 32;
constexpr uint32_t kCellEntries = 8;
// One cell, 3 x uint4: [ids 0-3 (u16), bounds 1, 2], [ids 4-7, bounds 3, 4],
// [bounds 5-7, bound of the first object left out].  The first vector is all
// a query reads when its hint is the cell's first entry and the second is
// farther than the best; bound 0 is never needed (entry 0's box is tested).
constexpr uint32_t kCellWords = 12;
constexpr __host__ __device__ uint32_t cell_id_word(uint32_t k) { return (k >> 1) + (k >= 4 ? 2u : 0u); }
constexpr __host__ __device__ uint32_t cell_bound_word(uint32_t k) { return k + (k < 3 ? 1u : 3u); }
// Leaf-order cache build (leafcache.cu) from the staged march scene.
struct LeafCacheLaunch {
    const float4* march_scene;  // object records on the device
    uint32_t n;                 // objects
    cudaTextureObject_t atlas;
    int sdf_f16;
    const void* sdf_cells;  // corner cells of the field meshes (dev_sdf.cuh), or null
    irtd::FieldFilter field_filter;
    float grid_org[3], grid_size[3];  // as the march reads them
    float margin;               // f32 error of a distance and of a point's place in its cell
    uint32_t* cells;            // kGridRes^3 * kCellWords words
};
cudaError_t irt_launch_leaf_cache(const LeafCacheLaunch& L, cudaStream_t st);
constexpr uint32_t kMaxBoundObjects = 256;  // distance bounds for scenes up to this many objects, else box bounds

struct SvgfLaunch {
    const irt_frame* frame;
    irt_gbuffer gbuffer;
    const float* old_depth;
    const void* old_normal;
    const void* in;          // temporal: noisy; variance/atrous: input radiance
    const void* aux;         // temporal: old radiance (feedback)
    const void* moments_in;  // temporal: old moments; variance: current moments
    void* out;
    void* out2;              // atrous: optional second output
    void* moments_out;       // temporal: current moments
    int step;
    int radiance_f16;
    int moments_f16;          // moments: 0 float4 (E[l], E[l^2], age, 0); 1 MomF16 (half mean, half deviation, f32 age)
    const float4* guide;      // per-pixel positions of this frame (or null)
    const float4* old_guide;  // ... of the previous frame (or null)
    const float4* feat;       // per-pixel edge-stopping features (or null)
    int after_guides;         // stage 0: the launch before this one was stage 6
    float4* old_guide_out;    // stage 6: also the guide of the previous frame's pixels (or null)
};
// irt_launch_svgf stages: 0 temporal, 1 variance, 2 a-trous, 5 depth and
// normal history (out = previous depth, out2 = previous normal), 6 position
// guide of this frame (out = float4[W*H]) and its edge-stopping features (out2 =
// float4[2*W*H]), and with old_guide_out the guide of the previous frame's
// pixels from old_depth and previous_inv_vp.

// VPL paths of one frame (vplgen.cu): lights on the device, ray casts
// against a workload's primitive table.
struct VplLaunch {
    const irt_frame* frame;
    irt::PrimTable prims;
    const irt_light* lights;
    irt_vpl* out;
};
cudaError_t irt_launch_vpls(const VplLaunch& L, cudaStream_t st);
// The workload's flattened primitive table and triangle tables on the
// current device (built on first use and kept with the workload).
cudaError_t irt_workload_prims(const irt_workload* wl, irt::PrimTable* out);

cudaError_t irt_launch_lighting(const LightingLaunch& L, int stage, cudaStream_t st);

// Corner cells of one field mesh (sdfcells.cu): records [base, base +
// (res-1)^3) of `out` from the atlas tile at `origin` (DevScene::sdf_cells).
cudaError_t irt_pack_sdf_cells(cudaTextureObject_t atlas, int f16, const uint32_t origin[3], uint32_t res,
                               uint64_t base, void* out, cudaStream_t st);
// sample_field of the mesh `row` (its device row values: hi[3] = first
// corner cell) at n grid-space points q (3 floats each); out: n floats.
namespace irtd {
struct DevScene;
}
cudaError_t irt_launch_sample_field(const irtd::DevScene& sc, const irt_mesh& row, const float* q, uint32_t n,
                                    float* out, cudaStream_t st);

// ------------------------------------------------------------------ batched views
// One launch per pass over the views of a batch.  `table` is a device array
// of n per-view argument records of the stage (lighting: the LightArgs of
// irt_lighting_args_fill; SVGF: the records of irt_svgf_view_fill),
// `frames` the n per-view frames on the device, `tile_start` n+1 block
// offsets (2-D kernels: tiles of bx x by pixels; 1-D kernels: 256 pixels).
struct BatchLaunch {
    uint32_t n;
    const irt_frame* frames;
    const void* table;
    const uint32_t* tile_start;
    uint32_t tiles;
    uint32_t bx, by;
    int gbuffer_format;
    int radiance_f16, moments_f16;
    int keep;
    int step;  // a-trous: 1 << iteration
};
size_t irt_lighting_args_size(int gbuffer_format);
void irt_lighting_args_fill(const LightingLaunch& L, void* out);
cudaError_t irt_launch_lighting_batched(const BatchLaunch& B, int stage, cudaStream_t st);
// SVGF stages of a batch: 0 temporal, 1 variance, 2 a-trous (BatchLaunch::
// step), 4 guides of the previous frame, 5 depth and normal history copy, 6
// guides and features of this frame.
size_t irt_svgf_view_size(int gbuffer_format);
void irt_svgf_view_fill(const SvgfLaunch& L, void* out);
cudaError_t irt_launch_svgf_batched(const BatchLaunch& B, int stage, cudaStream_t st);
cudaError_t irt_launch_svgf_spatial_batched(const BatchLaunch& B, int stage, cudaStream_t st);

// Batched march: views grouped by scene; each group's compact scene is
// staged in shared memory once per CTA and the group's ray queues (one per
// view) are consumed in order.
struct MarchQueue {
    RaySetup setup;
    const irt_frame* frame;  // the view's entry of the batch's device frame table
    uint32_t width, height;
};
struct alignas(16) MarchGroup {
    irt_frame f;                // counts[3] and sdf[] of the group's views
    const irt_object* objects;
    const irt_mesh* meshes;
    const irt_node* nodes;
    cudaTextureObject_t atlas;
    int sdf_f16;
    const void* sdf_cells;  // corner cells of the field meshes (dev_sdf.cuh), or null
    irtd::FieldFilter field_filter;
    uint32_t* error;
    const float4* march_scene;
    uint32_t scene_vec4;
    const uint4* cells;
    float grid_org[3], grid_inv[3], grid_size[3], grid_slack;
    uint32_t q_begin, q_end;    // the group's queues in the queue table
};
// Groups of one march launch, its kernel parameter (a batch of more launches again).
constexpr uint32_t kMarchGroups = 16;
struct MarchGroups {
    MarchGroup g[kMarchGroups];
    uint32_t n;
};
static_assert(sizeof(MarchGroups) <= 32764 - sizeof(void*), "kernel parameters of sm_70 and later");
struct MarchBatch {
    uint32_t n_groups;
    const MarchGroup* groups;   // device
    const MarchGroup* host_groups;
    const MarchQueue* queues;   // device
    uint32_t max_scene_bytes;
    int num_sms;
    int blocks_per_sm;          // 0 = occupancy maximum
    int fast;
    int sampler;                // march_sampler() of every group, or 3 where they differ
};
// Which build of the march kernel a scene's fields take: point-sampled f32 (0)
// or f16 (1) corner cells, or the filtered atlas (2, f32 only).
inline int march_sampler(const irtd::FieldFilter& filter, int sdf_f16) { return filter.linear ? 2 : sdf_f16 ? 1 : 0; }
cudaError_t irt_launch_ray_pools_batched(const MarchBatch& M, cudaStream_t st);
cudaError_t irt_launch_march_batched(const MarchBatch& M, cudaStream_t st);
// Lights with the spot direction normalised and cos(angle / 2) in
// direction_angle, the form the lighting kernels read.
cudaError_t irt_launch_prepare_lights(const irt_light* lights, uint32_t n, irt_light* out, cudaStream_t st);
cudaError_t irt_launch_svgf(const SvgfLaunch& L, int stage, cudaStream_t st);
// Stages 1 (variance) and 2 (a-trous), the fast-math SVGF passes.
cudaError_t irt_launch_svgf_spatial(const SvgfLaunch& L, int stage, cudaStream_t st);
