// march.cu — soft-shadow visibility of the frame's rays: ray set-up and a
// persistent march over the ray queue.
//
// visibility() of sdf.wgsl:61-81 is a clearance query at the surface point,
// for VPL rays one at the endpoint, then up to sdf_max_steps march steps, each
// a scene_distance query.  The first two do not depend on the ray: a pixel's
// two rays leave the same surface point, and all rays to a VPL share its
// endpoint.  So they run once per pixel and once per VPL, in coherent kernels
// of their own (ray_pools_kernel, ray_setup_kernel), with the same operations
// on the same operands, and the persistent march holds march steps only.  It
// restates them as a per-lane state machine; lanes that finish their rays
// refill together from their warp's reserved slice of the queue.  The march
// is bound by instruction issue under divergence (79 % issue active, DRAM
// idle) and the latency of the field's corner cells, so what counts is lanes
// per instruction, instructions, and resident warps.  Per 1920x1200 frame (24
// meshes, f32, set-up included): clearances and endpoints as phases of the
// march 3.22 ms at 14 lanes an instruction; as kernels of their own, and the
// march's stages rejoined by __syncwarp (lane_step), 2.42 ms at 19.4 lanes,
// of which the set-up is 0.14 ms; leaf bounds taken at the query point
// (leafcache.cu; 1.31 -> 1.13 evaluations a query, fewer entries tested)
// 2.11; short divides, flushed denormals, 256-bit cell loads 2.05; the cell
// found anew per candidate search instead of kept, 1.98; 36 warps 1.89; a
// kernel per field sampler 1.84; rays sorted by end (ray_setup_block) 1.68.
//
// scene_distance (sdf.wgsl:42-60) returns the minimum object distance: the
// walk skips a subtree only when its box bound exceeds the current best, and
// every object's distance is at least the distance to its BVH leaf box (the
// leaf box bounds the padded SDF box, which bounds the geometry box the
// distance is clamped to).  So visiting the same leaves in another order and
// skipping those whose box bound exceeds the current best yields the same
// best, the same closest object (ties aside) and the same voxel.  The march
// visits leaves in the order of a per-frame leaf-order cache (leafcache.cu):
// for the grid cell holding the query point, the leaves sorted by a lower
// bound of their distance from the cell's centre, stopping at the first whose
// bound exceeds the best so far plus the point's distance from the centre.
// Points outside the grid, or past the cached entries, test every leaf.
// Per object the arithmetic is object_distance()'s, evaluated on records
// staged in shared memory.
//
// The loop is flattened to one object per lane and iteration (see Query):
// lanes at different stages of their queries evaluate objects together.
//
// This file is built twice: as is (IEEE division and square root, the
// arithmetic of the per-pixel visibility()), and through march_fast.cu with
// approximate division and square root for the default fast march.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "dev_sdf.cuh"
#include "kernels.h"

#ifndef IRT_MARCH_FAST
#define IRT_MARCH_FAST 0
#endif

namespace irtd {
#if IRT_MARCH_FAST
namespace fast {
#else
namespace exact {
#endif

// Resident warps, set-up and march at 1920x1200: the single-view march at 56
// registers in CTAs of 192 threads, 6 per SM (36 warps, no spills), 1.89 ms;
// 4 CTAs of 256 (64 registers, 32 warps) 1.98, 5 (48 registers, spills) 2.14,
// 6 (40 registers) 2.47, 3 (24 warps) 2.39 before the query was slimmed.
constexpr int kMarchThreads = 192;
constexpr int kMarchCtasPerSm = 6;
// Queue entries a warp reserves per atomic (one per lane): the queue counter
// then sees one atomic per ~30 warp iterations instead of about one per
// iteration (1920x1200 room: 3.51 -> 3.43 ms with the L2 prefetch of the
// reserved records, 3.46 without; 64 entries 3.45 ms).
constexpr uint32_t kRayChunk = 32;
constexpr uint32_t kNone = 0xffffffffu;

struct Grid {
    const uint4* cells;
    float ox, oy, oz, ix, iy, iz;
    float sx, sy, sz;  // cell size
    float slack;       // error of an evaluated distance (Query::others)
};

// A distance query.  Its candidates are the hint object first (the previous
// closest, as scene_distance seeds it), then the leaf-order cache entries of
// the query point's cell that survive the walk's pruning tests (stopping at
// the first entry whose bound exceeds the best), then every leaf when the
// cached entries may not hold the minimum or the point is outside the grid.
// The march runs the queries of a warp's lanes as one flattened loop, one
// object per lane and iteration, so the evaluations of lanes at different
// stages (a hint, a second leaf) issue together; per query the candidates and
// their order are the same as a walk of one query at a time, so the results
// are too.
struct Query {
    float best;
    uint32_t closest, hint;
    uint32_t oid;  // the object to evaluate next, or kNone
    uint32_t cur;  // the candidate after it: 0..7 cache entries, 8 after them, >= kAll all leaves
    // Lower bound of the distance of every object but the closest.  Positive
    // distances are 1-Lipschitz (leafcache.cu), so a march step of length h
    // takes h (and the f16 and filter errors) off it, and a query whose hint is
    // nearer than that is complete without a look at the cache: most steps
    // near a ray's ends.  160x100 rays 129 -> 110 us, 480x300 247 -> 207; at full
    // size, where other lanes of the warp search anyway, within 1 %.
    float others;
};
constexpr uint32_t kAll = 16;

__device__ __forceinline__ void query_begin(Query& qy, uint32_t hint, uint32_t n, float others) {
    qy.others = others;
    qy.best = 1e20f;
    qy.closest = hint;
    qy.hint = hint;
    qy.cur = 0u;
    qy.oid = hint < n ? hint : kNone;
}

// The cache cell of a point (or kNone outside the grid) and the point's
// distance from the cell's centre.
__device__ __forceinline__ uint32_t cell_of(const Grid& g, V3 p, float& off_centre) {
    static_assert((kGridRes & (kGridRes - 1)) == 0, "the inside test takes the or of the three coordinates");
    const V3 f = {(p.x - g.ox) * g.ix, (p.y - g.oy) * g.iy, (p.z - g.oz) * g.iz};
    const V3 m = {__fadd_rd(f.x, kFloorMagic), __fadd_rd(f.y, kFloorMagic), __fadd_rd(f.z, kFloorMagic)};
    const uint32_t x = __float_as_uint(m.x) - kFloorBits, y = __float_as_uint(m.y) - kFloorBits,
                   z = __float_as_uint(m.z) - kFloorBits;
    const float half = kFloorMagic - .5f;  // m - half = the cell's centre; exact
    const V3 r = {(f.x - (m.x - half)) * g.sx, (f.y - (m.y - half)) * g.sy, (f.z - (m.z - half)) * g.sz};
    off_centre = sqrtf(dot(r, r));
    return (x | y | z) < kGridRes ? (z * kGridRes + y) * kGridRes + x : kNone;
}

// The walk's pruning test of an object's leaf box against the best so far.
__device__ __forceinline__ bool leaf_may_hold_best(const MObj& o, V3 p, float bound, float& others) {
    V3 delta = fmax3(fmax3(xyz(o.leaf_lo) - p, p - xyz(o.leaf_hi)), V3{0.f, 0.f, 0.f});
    V3 lb = delta * .9998f;
    const float d2 = dot(lb, lb);
    if (!(d2 > bound * bound)) return true;
    others = fminf(others, sqrtf(d2));
    return false;
}

// Next object to evaluate for the query at p, or kNone when it is complete.
// The cell is found anew on each call (1.13 a query): kept in the query, it
// and the point would live through the evaluation.
__device__ __forceinline__ uint32_t query_next(Query& qy, V3 p, const Grid& g, const MObj* objs, uint32_t n,
                                               uint32_t* err) {
    const float bound = fmaxf(qy.best, 0.f);
    if (qy.cur == 0u) {
        if (bound <= qy.others) return kNone;
        qy.others = 1e20f;
    }
    float off_centre;
    const uint32_t cell = cell_of(g, p, off_centre);
    const float reach = bound + off_centre;
    // the objects from a cache entry on lie beyond the query's reach
    auto rest = [&](float b) {
        if (!(b > reach)) return false;
        qy.others = fminf(qy.others, b - off_centre);
        return true;
    };
    const uint32_t* cw = reinterpret_cast<const uint32_t*>(g.cells) + (size_t)cell * kCellWords;
    uint32_t c = qy.cur;
    if (cell == kNone) {
        if (c == 0u) c = kAll;
    } else if (c == 0u) {  // usually the hint is the cell's first entry and the second one is farther
        const uint4 w = __ldg(reinterpret_cast<const uint4*>(cw));
        if ((w.x & 0xffffu) == qy.hint) {
            if (rest(__uint_as_float(w.z))) return kNone;
            c = 1u;
        }
    }
    for (;; c++) {
        uint32_t oid;
        if (c < kCellEntries) {
            if (c > 0u && rest(__uint_as_float(__ldg(cw + cell_bound_word(c))))) return kNone;
            oid = (__ldg(cw + cell_id_word(c)) >> ((c & 1u) * 16u)) & 0xffffu;
            if (oid == 0xffffu) return kNone;
            if (!index_ok(err, oid, n)) continue;
        } else if (c < kAll) {  // every cached entry fits: the ones left out may too
            if (rest(__uint_as_float(__ldg(cw + cell_bound_word(kCellEntries))))) return kNone;
            c = kAll - 1u;
            continue;
        } else {
            oid = c - kAll;
            if (oid >= n) return kNone;
        }
        if (oid != qy.hint && leaf_may_hold_best(objs[oid], p, bound, qy.others)) {
            qy.cur = c + 1u;
            return oid;
        }
    }
}

// Object `oid`'s distance folded into the query (the hint sets the best
// unconditionally, as scene_distance seeds it).
__device__ __forceinline__ void query_eval(Query& qy, V3 p, const DevScene& sc, const MObj* objs, uint32_t oid) {
    const float d = object_distance(sc, p, objs[oid]);
    qy.others = fminf(qy.others, fmaxf(d, qy.best));  // the farther of the two (best is 1e20 before the first)
    if (oid == qy.hint || d < qy.best) {
        qy.best = d;
        qy.closest = oid;
    }
}

// One distance query from p without a hint, walked to its end: the nearest
// object, or kNone.
__device__ __forceinline__ uint32_t query_closest(const DevScene& sc, const Grid& g, const MObj* objs, uint32_t n,
                                                  V3 p) {
    Query qy;
    query_begin(qy, kNone, n, -1.f);
    for (;;) {
        const uint32_t oid = query_next(qy, p, g, objs, n, sc.error);
        if (oid == kNone) break;
        query_eval(qy, p, sc, objs, oid);
    }
    return qy.closest;
}

// The scene as a kernel's CTA reads it.
struct SceneRefs {
    const MObj* objs;
    uint32_t n_obj;
    float eps;
    uint32_t max_steps;
};
__device__ __forceinline__ SceneRefs scene_refs(const irt_frame& f, const float4* smem) {
    return SceneRefs{reinterpret_cast<const MObj*>(smem), f.counts[3], f.sdf[1], to_u32(f.sdf[0])};
}

// A point moved off the surface along its normal (sdf.wgsl:63, :66).
__device__ __forceinline__ V3 cleared(V3 p, V3 n, uint32_t closest, const SceneRefs& R) {
    const float voxel = closest < R.n_obj ? R.objs[closest].meta.y : R.eps;
    return p + n * clearance_epsilon(R.eps, voxel);
}

// March endpoint of a VPL: cleared, when it has a normal.
__device__ __forceinline__ V3 vpl_endpoint(const DevScene& sc, const Grid& g, const SceneRefs& R, V3 pos, V3 nrm) {
    if (!(dot(nrm, nrm) > .5f)) return pos;
    return cleared(pos, nrm, query_closest(sc, g, R.objs, R.n_obj, pos), R);
}

__device__ __forceinline__ const irt_vpl* pool_vpl(const RaySetup& s, uint32_t v) {
    const uint32_t n = s.vpl_count;
    return v < n ? s.cur + v : v < 2u * n ? s.prev + (v - n) : s.arch + (v - 2u * n);
}

// VPL archive slot frame % slots (src/renderer.rs:1873-1884), the queue's
// reset, and every VPL's march endpoint: entry v of the frame's pools.
__device__ __forceinline__ void ray_pool_entry(const RaySetup& s, const DevScene& sc, const Grid& g,
                                               const SceneRefs& R, uint32_t frame_index, uint32_t v) {
    const uint32_t n = s.vpl_count, first = (2u + frame_index % s.slots) * n;
    const bool fresh = v >= first && v < first + n;  // the archive slot this frame's pool goes to
    const float4* src = reinterpret_cast<const float4*>(fresh ? s.cur + (v - first) : pool_vpl(s, v));
    const float4 pos = __ldg(src), nrm = __ldg(src + 1);
    if (fresh) {
        float4* dst = reinterpret_cast<float4*>(s.arch + (v - 2u * n));
        dst[0] = pos;
        dst[1] = nrm;
        dst[2] = __ldg(src + 2);
    }
    if (s.ends) {
        const V3 e = vpl_endpoint(sc, g, R, xyz(pos), xyz(nrm));
        s.ends[v] = make_float4(e.x, e.y, e.z, 0.f);
    }
}

// The ray set-up of a block's 32x16 pixels (a warp takes 8x4 of them): each
// pixel's clearance, the begin of its rays' marches, and their records
// appended to the queue, the block's rays of a class sorted by where they end
// (one atomic per class and block).  The pixels of a block see nearly the same
// point, so rays to neighbouring ends stay together all the way and the
// march's warps meet the same objects: march 1.72 -> 1.55 ms at 1920x1200 f32,
// the set-up itself 0.145 -> 0.133 (latency of its dependent reads; blocks of
// 1024 pixels give the march nothing more, bins by start object 1.56).  VPL
// rays fill the queue from the front and light rays from the back (ray_slot),
// so the march takes whole runs of one class; each ray's result slot is in its
// record, so the order changes no result.  Rays resolved without a march step
// write their visibility here.
constexpr uint32_t kSetupThreads = 512, kSetupW = 32, kSetupH = 16;
constexpr uint32_t kEndBins = 512;  // 8x8x8 over the cache grid, in Morton order
struct SetupShared {
    uint32_t bins[kEndBins];  // rays per end: VPL rays in the low half, light rays in the high half
    uint32_t warp_total[kSetupThreads / 32];
    uint32_t base[2];
};
static_assert(kEndBins == kSetupThreads, "one bin a thread in the scan");

__device__ __forceinline__ uint32_t end_bin(const Grid& g, V3 p) {
    auto axis = [](float f) {  // 0..7, spread to every third bit
        const uint32_t c = (uint32_t)fminf(fmaxf(f, 0.f), (float)(kGridRes - 1)) / (kGridRes / 8);
        return (c & 1u) | (c & 2u) << 2 | (c & 4u) << 4;
    };
    return axis((p.x - g.ox) * g.ix) | axis((p.y - g.oy) * g.iy) << 1 | axis((p.z - g.oz) * g.iz) << 2;
}

__device__ __forceinline__ void ray_setup_block(const RaySetup& s, const DevScene& sc, const Grid& g,
                                                const SceneRefs& R, uint32_t W, uint32_t H, uint32_t tile,
                                                SetupShared& sh) {
    const unsigned full = 0xffffffffu;
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t / 32u;
    const uint32_t across = (W + kSetupW - 1) / kSetupW;
    const uint32_t x = (tile % across) * kSetupW + (warp & 3u) * 8u + (lane & 7u);
    const uint32_t y = (tile / across) * kSetupH + (warp >> 2) * 4u + (lane >> 3);
    const uint32_t i = y * W + x;
    __syncthreads();  // the previous tile's bins are read
    sh.bins[t] = 0u;
    __syncthreads();
    uint32_t light = kNoRay, vpl = kNoRay, hint = kNone, bin_d = 0, bin_v = 0, rank_d = 0, rank_v = 0;
    MarchState d, v;
    if (x < W && y < H) {
        const float4 prep = load_written(s.prep + i);
        light = __float_as_uint(prep.w);
        vpl = load_written(s.prep_vpl + i);
        if (light != kNoRay || vpl != kNoRay) {
            const V3 p = xyz(__ldg(s.guide + i));
            hint = query_closest(sc, g, R.objs, R.n_obj, p);
            d.origin = cleared(p, xyz(prep), hint, R);
            v.origin = d.origin;
        }
        if (light != kNoRay) {
            const V3 end = xyz(__ldg(reinterpret_cast<const float4*>(s.lights + light)));
            const float out = march_begin(d, end, R.eps, R.max_steps);
            if (out >= 0.f) {
                s.vis[2 * (size_t)i] = out;
                light = kNoRay;
            } else {
                bin_d = end_bin(g, end);
                rank_d = atomicAdd(&sh.bins[bin_d], 1u << 16) >> 16;
            }
        }
        if (vpl != kNoRay) {
            V3 end;
            if (s.ends) {
                end = xyz(__ldg(s.ends + vpl));
            } else {
                const float4* src = reinterpret_cast<const float4*>(pool_vpl(s, vpl));
                end = vpl_endpoint(sc, g, R, xyz(__ldg(src)), xyz(__ldg(src + 1)));
            }
            const float out = march_begin(v, end, R.eps, R.max_steps);
            if (out >= 0.f) {
                s.vis[2 * (size_t)i + 1] = out;
                vpl = kNoRay;
            } else {
                bin_v = end_bin(g, end);
                rank_v = atomicAdd(&sh.bins[bin_v], 1u) & 0xffffu;
            }
        }
    }
    __syncthreads();
    // Exclusive prefix sums of both classes at once (at most 512 rays each).
    const uint32_t own = sh.bins[t];
    uint32_t sum = own;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t up = __shfl_up_sync(full, sum, o);
        if (lane >= o) sum += up;
    }
    if (lane == 31u) sh.warp_total[warp] = sum;
    __syncthreads();
    uint32_t before = 0;
#pragma unroll
    for (uint32_t k = 0; k < kSetupThreads / 32; k++) before += k < warp ? sh.warp_total[k] : 0u;
    sh.bins[t] = before + sum - own;
    if (t == kSetupThreads - 1) {
        const uint32_t total = before + sum;
        sh.base[0] = total & 0xffffu ? atomicAdd(s.counters, total & 0xffffu) : 0u;
        sh.base[1] = total >> 16 ? atomicAdd(s.counters + 2, total >> 16) : 0u;
    }
    __syncthreads();
    const uint32_t cap = 2u * W * H;
    auto emit = [&](const MarchState& m, uint32_t at, uint32_t slot) {
        if (!index_ok(sc.error, at, cap)) return;
        s.rays[at].a = make_float4(m.origin.x, m.origin.y, m.origin.z, __uint_as_float(slot));
        s.rays[at].b = make_float4(m.dir.x, m.dir.y, m.dir.z, m.limit);
        s.hints[at] = (uint16_t)hint;
    };
    if (vpl != kNoRay) emit(v, sh.base[0] + (sh.bins[bin_v] & 0xffffu) + rank_v, 2u * i + 1u);
    if (light != kNoRay) emit(d, cap - 1u - (sh.base[1] + (sh.bins[bin_d] >> 16) + rank_d), 2u * i);
}

// A warp's reserved slice [next, end) of a ray queue; `drained` once the
// queue counter has passed the queue's end.  Warp-uniform.
struct RaySlice {
    uint32_t next, end;
    bool drained;
};

// Queue indices for the warp's idle lanes (`need`, a ballot): this lane's
// index, or n_rays for none.  The slice is used first; a new reservation
// takes kRayChunk entries while more than `keep` entries are left (two
// chunks per warp of the grid: the warp's own slice end trails the counter
// by up to one), else what the idle lanes still need.  The lanes prefetch a
// new chunk's records into L2, so the loads of the lanes that take them
// later hit L2 instead of DRAM.
__device__ __forceinline__ uint32_t slice_take(RaySlice& s, unsigned need, uint32_t* counter, uint32_t n_rays,
                                               uint32_t keep, int lane, const RayRecord* rays, uint32_t front,
                                               uint32_t cap) {
    const unsigned full = 0xffffffffu;
    const uint32_t cnt = (uint32_t)__popc(need);
    const uint32_t avail = s.end - s.next;
    const uint32_t rank = (uint32_t)__popc(need & ((1u << lane) - 1u));
    uint32_t idx = rank < avail ? s.next + rank : n_rays;
    if (avail >= cnt) {
        s.next += cnt;
    } else if (s.drained) {
        s.next = s.end;
    } else {
        const uint32_t want = s.end + keep < n_rays ? kRayChunk : cnt - avail;
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(counter, want);
        base = __shfl_sync(full, base, 0);
        if (rank >= avail) idx = base + (rank - avail);
        if (base >= n_rays) {
            s.drained = true;
            s.next = s.end = 0;
        } else {
            if ((uint32_t)lane < want && base + (uint32_t)lane < n_rays) {
                const uint32_t slot = ray_slot(base + (uint32_t)lane, front, cap);
                if (slot < cap) asm volatile("prefetch.global.L2 [%0];" ::"l"(rays + slot));
            }
            s.drained = base + want >= n_rays;
            s.end = s.drained ? n_rays : base + want;
            s.next = min(base + (cnt - avail), s.end);
        }
    }
    return idx;
}

// One lane's ray and the query of its current march step.
struct Lane {
    MarchState m;
    Query qy;
    uint32_t slot;
    bool active;
};
__device__ __forceinline__ void lane_reset(Lane& L) {
    L.m.closest = kNone;
    L.m.origin = V3{0.f, 0.f, 0.f};
    L.m.dir = V3{0.f, 0.f, 0.f};
    L.m.t = L.m.limit = 0.f;
    L.m.result = 1.f;
    L.m.previous = 1e20f;
    L.m.step = 0;
    L.qy.oid = kNone;
    L.active = false;
}
// The ray of record `at`, as ray_setup_block left it, and its first query.
__device__ __forceinline__ void lane_take(Lane& L, const RaySetup& s, uint32_t at, const SceneRefs& R) {
    const float4* r = reinterpret_cast<const float4*>(s.rays + at);
    const float4 a = load_written(r), b = load_written(r + 1);
    const uint32_t hint = load_written(s.hints + at);
    L.m.origin = V3{a.x, a.y, a.z};
    L.m.dir = V3{b.x, b.y, b.z};
    L.m.limit = b.w;
    L.m.t = R.eps;
    L.m.result = 1.f;
    L.m.previous = 1e20f;
    L.m.step = 0;
    L.m.closest = hint;
    L.slot = __float_as_uint(a.w);
    L.active = true;
    query_begin(L.qy, hint, R.n_obj, -1.f);
}
// One iteration of a warp's lanes, stage by stage: every active lane
// evaluates its query's object; finds the next one; and where the query has
// none left, completes its march step (sdf.wgsl:68-80) and begins the ray's
// next query with its hint.  The lanes meet after each stage: without the
// __syncwarp the compiler keeps lanes that took different ways through the
// candidate search apart through the next evaluation (14.1 against 19.4 lanes
// an instruction, 760 against 531 million warp instructions at 960x600).
__device__ __forceinline__ void lane_step(Lane& L, const DevScene& sc, const Grid& grid, const SceneRefs& R, float k,
                                          float* vis, uint32_t cap) {
    if (L.active && L.qy.oid != kNone) query_eval(L.qy, march_point(L.m), sc, R.objs, L.qy.oid);
    __syncwarp();
    if (L.active) L.qy.oid = query_next(L.qy, march_point(L.m), grid, R.objs, R.n_obj, sc.error);
    __syncwarp();
    if (L.active && L.qy.oid == kNone) {
        L.m.closest = L.qy.closest;
        const float out = march_after(L.m, L.qy.best, R.eps, k, R.max_steps);
        if (out >= 0.f) {
            if (index_ok(sc.error, L.slot, cap)) vis[L.slot] = out;
            L.active = false;
        } else {
            query_begin(L.qy, L.m.closest, R.n_obj, L.qy.others * .997f - (L.qy.best + grid.slack));
        }
    }
    __syncwarp();
}

// The march kernels are built per field sampler, so that each carries the
// registers and branches of one (march 1.77 -> 1.70 ms at 1920x1200 f32); a
// batch whose scenes differ runs the one that tests per scene.
enum Sampler : int { kPointF32 = 0, kPointF16 = 1, kLinearF32 = 2, kAnySampler = 3 };
// CTAs of the batched march: as the single-view kernel's, but the one for any
// sampler, which would spill at 56 registers.
constexpr int march_threads(int sampler) { return sampler == kAnySampler ? 128 : kMarchThreads; }
constexpr int march_ctas(int sampler) { return sampler == kAnySampler ? 8 : kMarchCtasPerSm; }
template <int S>
__device__ __forceinline__ void assume_sampler(DevScene& sc) {
    if (S == kPointF32 || S == kPointF16) sc.filter.linear = 0;
    if (S == kLinearF32) __builtin_assume(sc.filter.linear != 0);
    if (S != kAnySampler) sc.sdf_f16 = S == kPointF16;
}

// Idle lanes a warp collects before it refills them, so that the refill's
// instructions run for several lanes at once: 1 lane 2.49 ms, 3 or 6 lanes
// 2.43, 10 lanes 2.49, 16 lanes 2.68 (set-up and march at 1920x1200).
constexpr int kRefill = 6;
constexpr uint32_t kMinLanes = 4;

__global__ void __launch_bounds__(kMarchThreads) ray_pools_kernel(const __grid_constant__ irt_frame f, const DevScene sc,
                                                                  const float4* __restrict__ march_scene,
                                                                  uint32_t scene_vec4, const Grid grid,
                                                                  const __grid_constant__ RaySetup setup) {
    extern __shared__ float4 smem[];
    for (uint32_t i = threadIdx.x; i < scene_vec4; i += blockDim.x) smem[i] = __ldg(march_scene + i);
    frame_kernel_begin();  // the records above are not the frame's to write
    __syncthreads();
    const SceneRefs R = scene_refs(f, smem);
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < 4) setup.counters[t] = 0u;
    const uint32_t n = (setup.slots + 2u) * setup.vpl_count;
    for (uint32_t v = t; v < n; v += gridDim.x * blockDim.x) ray_pool_entry(setup, sc, grid, R, f.size[2], v);
}

__global__ void __launch_bounds__(kSetupThreads, 2) ray_setup_kernel(const __grid_constant__ irt_frame f, const DevScene sc,
                                                                  const float4* __restrict__ march_scene,
                                                                  uint32_t scene_vec4, const Grid grid,
                                                                  const __grid_constant__ RaySetup setup) {
    extern __shared__ float4 smem[];
    __shared__ SetupShared sh;
    for (uint32_t i = threadIdx.x; i < scene_vec4; i += blockDim.x) smem[i] = __ldg(march_scene + i);
    frame_kernel_begin();  // the records above are not the frame's to write
    __syncthreads();
    const SceneRefs R = scene_refs(f, smem);
    const uint32_t W = f.size[0], H = f.size[1];
    const uint32_t tiles = ((W + kSetupW - 1) / kSetupW) * ((H + kSetupH - 1) / kSetupH);
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) ray_setup_block(setup, sc, grid, R, W, H, t, sh);
}

template <int S>
__global__ void __launch_bounds__(kMarchThreads, kMarchCtasPerSm) march_kernel(const __grid_constant__ irt_frame f, DevScene sc,
                                                    const float4* __restrict__ march_scene, uint32_t scene_vec4,
                                                    const Grid grid, const __grid_constant__ RaySetup setup) {
    extern __shared__ float4 smem[];
    for (uint32_t i = threadIdx.x; i < scene_vec4; i += blockDim.x) smem[i] = __ldg(march_scene + i);
    frame_kernel_begin();  // the records above are not the frame's to write
    __syncthreads();
    assume_sampler<S>(sc);
    const SceneRefs R = scene_refs(f, smem);
    const uint32_t front = *(volatile uint32_t*)&setup.counters[0];
    const uint32_t n_rays = front + *(volatile uint32_t*)&setup.counters[2];
    const uint32_t cap = 2u * f.size[0] * f.size[1];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;

    // A queue shorter than the grid's lanes is spread over its warps, a few
    // lanes each: a step then runs fewer lanes' ways (160x100: 32 000 rays).
    const uint32_t warps = gridDim.x * (blockDim.x / 32u);
    const uint32_t lanes = min(max((n_rays + warps - 1u) / warps, kMinLanes), 32u);
    const unsigned mine = lanes == 32u ? full : (1u << lanes) - 1u;
    const int refill = min(kRefill, (int)lanes);

    bool exhausted = false;  // warp-uniform: the queue has no rays left
    Lane L;
    lane_reset(L);
    RaySlice slice{0u, 0u, false};
    const uint32_t keep = 2u * warps * kRayChunk;
    for (;;) {
        const unsigned idle = __ballot_sync(full, !L.active), need = idle & mine;
        if (exhausted) {
            if (idle == full) break;
        } else if (__popc(need) >= refill) {
            const uint32_t idx = slice_take(slice, need, &setup.counters[1], n_rays, keep, lane, setup.rays, front, cap);
            exhausted = slice.drained && slice.next >= slice.end;
            if ((need >> lane & 1u) && idx < n_rays && index_ok(sc.error, ray_slot(idx, front, cap), cap))
                lane_take(L, setup, ray_slot(idx, front, cap), R);
        }
        lane_step(L, sc, grid, R, f.sdf[2], setup.vis, cap);
    }
}

// ---------------------------------------------------------------- batched views
// For each scene group a CTA stages the group record and its compact scene in
// shared memory, then runs the single-view bodies over the group's views.
constexpr uint32_t kGroupVec4 = (uint32_t)((sizeof(MarchGroup) + 15) / 16);

// Stages group g into smem; its scene follows the record.
__device__ __forceinline__ const MarchGroup& stage_group(const MarchGroup* __restrict__ groups, uint32_t g,
                                                         float4* smem) {
    const MarchGroup& G = *reinterpret_cast<const MarchGroup*>(smem);
    __syncthreads();  // every warp is done with the previous group's records
    const float4* gsrc = reinterpret_cast<const float4*>(groups + g);
    for (uint32_t i = threadIdx.x; i < kGroupVec4; i += blockDim.x) smem[i] = __ldg(gsrc + i);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < G.scene_vec4; i += blockDim.x) smem[kGroupVec4 + i] = __ldg(G.march_scene + i);
    __syncthreads();
    return G;
}
__device__ __forceinline__ DevScene group_scene(const MarchGroup& G) {
    DevScene sc;
    sc.objects = G.objects;
    sc.meshes = G.meshes;
    sc.nodes = G.nodes;
    sc.lights = nullptr;
    sc.atlas = G.atlas;
    sc.sdf_f16 = G.sdf_f16;
    sc.sdf_cells = G.sdf_cells;
    sc.filter = G.field_filter;
    sc.error = G.error;
    return sc;
}
__device__ __forceinline__ Grid group_grid(const MarchGroup& G) {
    return Grid{G.cells,        G.grid_org[0],  G.grid_org[1],  G.grid_org[2],  G.grid_inv[0],
                G.grid_inv[1], G.grid_inv[2], G.grid_size[0], G.grid_size[1], G.grid_size[2], G.grid_slack};
}

__global__ void __launch_bounds__(128) ray_pools_batched_kernel(const MarchGroup* __restrict__ groups, uint32_t n_groups,
                                                                const MarchQueue* __restrict__ queues) {
    extern __shared__ float4 smem[];
    for (uint32_t g = 0; g < n_groups; g++) {
        const MarchGroup& G = stage_group(groups, g, smem);
        const DevScene sc = group_scene(G);
        const Grid grid = group_grid(G);
        const SceneRefs R = scene_refs(G.f, smem + kGroupVec4);
        // Entries of all the group's views in one run, so that small pools share the grid.
        uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
        if (t < 4)
            for (uint32_t q = G.q_begin; q < G.q_end; q++) queues[q].setup.counters[t] = 0u;
        for (uint32_t q = G.q_begin; q < G.q_end; q++) {
            const MarchQueue& Q = queues[q];
            const uint32_t n = (Q.setup.slots + 2u) * Q.setup.vpl_count;
            for (; t < n; t += gridDim.x * blockDim.x) ray_pool_entry(Q.setup, sc, grid, R, Q.frame->size[2], t);
            t -= n;
        }
    }
}

__global__ void __launch_bounds__(kSetupThreads, 2) ray_setup_batched_kernel(const MarchGroup* __restrict__ groups, uint32_t n_groups,
                                                            const MarchQueue* __restrict__ queues) {
    extern __shared__ float4 smem[];
    __shared__ SetupShared sh;
    for (uint32_t g = 0; g < n_groups; g++) {
        const MarchGroup& G = stage_group(groups, g, smem);
        const DevScene sc = group_scene(G);
        const Grid grid = group_grid(G);
        const SceneRefs R = scene_refs(G.f, smem + kGroupVec4);
        uint32_t t = blockIdx.x;
        for (uint32_t q = G.q_begin; q < G.q_end; q++) {
            const MarchQueue& Q = queues[q];
            const uint32_t tiles = ((Q.width + kSetupW - 1) / kSetupW) * ((Q.height + kSetupH - 1) / kSetupH);
            const RaySetup s = Q.setup;
            for (; t < tiles; t += gridDim.x) ray_setup_block(s, sc, grid, R, Q.width, Q.height, t, sh);
            t -= tiles;
        }
    }
}

// The march over a group's queues in order; a lane keeps its queue's index.
// The groups are a kernel parameter: a group's constants are then read where
// they are used, as the single-view kernel reads its own.  Copies from a record
// in shared memory lived in registers: 64 of them, 32 warps an SM; now 56 and
// 36 warps (8 views of 5.2 Mpixel, the whole frame 9208 -> 9162 us).
template <int S>
__global__ void __launch_bounds__(march_threads(S), march_ctas(S)) march_batched_kernel(const __grid_constant__ MarchGroups groups,
                                                                     const MarchQueue* __restrict__ queues) {
    extern __shared__ float4 smem[];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    for (uint32_t g = 0; g < groups.n; g++) {
        const MarchGroup& G = groups.g[g];
        __syncthreads();  // every warp is done with the previous group's records
        for (uint32_t i = threadIdx.x; i < G.scene_vec4; i += blockDim.x) smem[i] = __ldg(G.march_scene + i);
        __syncthreads();
        DevScene sc = group_scene(G);
        assume_sampler<S>(sc);
        const Grid grid = group_grid(G);
        const SceneRefs R = scene_refs(G.f, smem);
        uint32_t q = G.q_begin;
        bool exhausted = q >= G.q_end;
        uint32_t front = exhausted ? 0u : *(volatile const uint32_t*)&queues[q].setup.counters[0];
        uint32_t n_rays = exhausted ? 0u : front + *(volatile const uint32_t*)&queues[q].setup.counters[2];
        uint32_t lq = 0;
        Lane L;
        lane_reset(L);
        RaySlice slice{0u, 0u, false};
        const uint32_t keep = 2u * gridDim.x * (blockDim.x / 32u) * kRayChunk;
        for (;;) {
            const unsigned need = __ballot_sync(full, !L.active);
            if (exhausted) {
                if (need == full) break;
            } else if (__popc(need) >= kRefill) {
                const MarchQueue& Q = queues[q];
                const uint32_t cap = 2u * Q.width * Q.height;
                const uint32_t idx = slice_take(slice, need, &Q.setup.counters[1], n_rays, keep, lane, Q.setup.rays,
                                                front, cap);
                if (!L.active && idx < n_rays && index_ok(sc.error, ray_slot(idx, front, cap), cap)) {
                    lane_take(L, Q.setup, ray_slot(idx, front, cap), R);
                    lq = q;
                }
                if (slice.drained && slice.next >= slice.end) {  // this queue is used up: the next view's
                    slice = RaySlice{0u, 0u, false};
                    q++;
                    if (q >= G.q_end) exhausted = true;
                    else {
                        front = *(volatile const uint32_t*)&queues[q].setup.counters[0];
                        n_rays = front + *(volatile const uint32_t*)&queues[q].setup.counters[2];
                    }
                }
            }
            lane_step(L, sc, grid, R, G.f.sdf[2], queues[lq].setup.vis, 2u * queues[lq].width * queues[lq].height);
        }
    }
}

}  // namespace fast / exact
}  // namespace irtd

#if IRT_MARCH_FAST
#define IRT_MARCH_NS irtd::fast
#else
#define IRT_MARCH_NS irtd::exact
#endif

// The carveout (percent of the SM's shared-memory maximum) that holds
// `blocks` CTAs of `smem` dynamic bytes plus the runtime's per-CTA reserve,
// and no more: the rest of the unified storage stays L1, where the leaf-order
// cache cells and SDF corner records of the march hit (1920x1200 room:
// 3.555 -> 3.531 ms against the driver's own choice; 50 % measured 3.589).
static cudaError_t march_prefer_l1(const void* kernel, uint32_t smem, int blocks) {
    int device = 0, per_sm = 0, reserved = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, device);
    if (e != cudaSuccess) return e;
    if (per_sm <= 0) return cudaSuccess;
    const long long need = (long long)blocks * ((long long)smem + reserved);
    const int pct = (int)std::min(100LL, (need * 100 + per_sm - 1) / per_sm);
    return cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, pct);
}

namespace {

// A kernel's dynamic shared memory limit and its resident CTAs per SM for a
// scene's bytes.  The limit is the function's, shared by every thread that
// launches it on the device, so it is raised once to all a CTA can have and
// never follows a scene.  The carveout is a hint, set when the bytes change.
struct KernelFit {
    static constexpr int kDevices = 64, kSizes = 16;
    struct Device {
        bool raised;
        uint32_t carveout_for, next;
        uint32_t bytes[kSizes];  // 0: unused (no scene is empty)
        int per_sm[kSizes];
    };
    std::mutex mu;
    Device devices[kDevices] = {};

    cudaError_t set(const void* kernel, int threads, uint32_t bytes, int prefer_blocks, int& per_sm) {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        if (dev < 0 || dev >= kDevices) return cudaErrorInvalidDevice;
        std::lock_guard<std::mutex> lock(mu);
        Device& d = devices[dev];
        if (!d.raised) {
            int most = 0;
            cudaFuncAttributes own;
            e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
            if (e == cudaSuccess) e = cudaFuncGetAttributes(&own, kernel);
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         most - (int)own.sharedSizeBytes);
            if (e != cudaSuccess) return e;
            d.raised = true;
        }
        if (d.carveout_for != bytes) {
            e = march_prefer_l1(kernel, bytes, prefer_blocks);
            if (e != cudaSuccess) return e;
            d.carveout_for = bytes;
        }
        for (int k = 0; k < kSizes; k++)
            if (d.bytes[k] == bytes) {
                per_sm = d.per_sm[k];
                return cudaSuccess;
            }
        int fits = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fits, kernel, threads, bytes);
        if (e != cudaSuccess) return e;
        if (fits < 1) return cudaErrorInvalidConfiguration;
        const uint32_t k = d.next++ % kSizes;
        d.bytes[k] = bytes;
        d.per_sm[k] = per_sm = fits;
        return cudaSuccess;
    }
};

irtd::DevScene launch_scene(const MarchLaunch& M) {
    irtd::DevScene sc;
    sc.objects = M.objects;
    sc.meshes = M.meshes;
    sc.nodes = M.nodes;
    sc.lights = nullptr;
    sc.atlas = M.atlas;
    sc.sdf_f16 = M.sdf_f16;
    sc.sdf_cells = M.sdf_cells;
    sc.filter = M.field_filter;
    sc.error = M.error;
    return sc;
}
IRT_MARCH_NS::Grid launch_grid(const MarchLaunch& M) {
    return IRT_MARCH_NS::Grid{M.cells,        M.grid_org[0],  M.grid_org[1],  M.grid_org[2],  M.grid_inv[0],
                              M.grid_inv[1], M.grid_inv[2], M.grid_size[0], M.grid_size[1], M.grid_size[2], M.grid_slack};
}

}  // namespace

#if IRT_MARCH_FAST
#define IRT_MARCH_FN(name) name##_fast
#else
#define IRT_MARCH_FN(name) name##_exact
#endif

cudaError_t IRT_MARCH_FN(irt_launch_ray_pools)(const MarchLaunch& M, cudaStream_t st) {
    using namespace IRT_MARCH_NS;
    const uint32_t smem = irt_march_scene_bytes(M.frame->counts[3]);
    static KernelFit fit;
    int per_sm;
    cudaError_t e = fit.set((const void*)ray_pools_kernel, kMarchThreads, smem, 1, per_sm);
    if (e != cudaSuccess) return e;
    const uint32_t entries = (M.setup.slots + 2u) * M.setup.vpl_count;
    const uint32_t blocks = std::min((uint32_t)M.num_sms, (entries + kMarchThreads - 1) / kMarchThreads);
    return launch_behind(ray_pools_kernel, dim3(blocks), dim3(kMarchThreads), smem, st, *M.frame, launch_scene(M),
                         M.march_scene, smem / 16, launch_grid(M), M.setup);
}

cudaError_t IRT_MARCH_FN(irt_launch_march)(const MarchLaunch& M, cudaStream_t st) {
    using namespace IRT_MARCH_NS;
    const uint32_t smem = irt_march_scene_bytes(M.frame->counts[3]);
    typedef decltype(&march_kernel<kPointF32>) Kernel;
    static const Kernel kernels[] = {march_kernel<kPointF32>, march_kernel<kPointF16>, march_kernel<kLinearF32>};
    const int sampler = march_sampler(M.field_filter, M.sdf_f16);
    static KernelFit set_up, march[3];
    int set_up_per_sm, march_per_sm;
    cudaError_t e = set_up.set((const void*)ray_setup_kernel, kSetupThreads, smem, 2, set_up_per_sm);
    if (e == cudaSuccess)
        e = march[sampler].set((const void*)kernels[sampler], kMarchThreads, smem, kMarchCtasPerSm, march_per_sm);
    if (e != cudaSuccess) return e;
    const irtd::DevScene sc = launch_scene(M);
    const Grid g = launch_grid(M);
    e = launch_behind(ray_setup_kernel, dim3(M.num_sms * set_up_per_sm), dim3(kSetupThreads), smem, st, *M.frame, sc,
                      M.march_scene, smem / 16, g, M.setup);
    if (e != cudaSuccess) return e;
    return launch_behind(kernels[sampler], dim3(M.num_sms * march_per_sm), dim3(kMarchThreads), smem, st, *M.frame, sc,
                         M.march_scene, smem / 16, g, M.setup);
}

cudaError_t IRT_MARCH_FN(irt_launch_ray_pools_batched)(const MarchBatch& M, cudaStream_t st) {
    using namespace IRT_MARCH_NS;
    if (M.n_groups == 0) return cudaSuccess;
    const uint32_t smem = kGroupVec4 * 16 + M.max_scene_bytes;
    static KernelFit fit;
    int per_sm;
    cudaError_t e = fit.set((const void*)ray_pools_batched_kernel, 128, smem, 1, per_sm);
    if (e != cudaSuccess) return e;
    ray_pools_batched_kernel<<<M.num_sms * std::min(per_sm, 2), 128, smem, st>>>(M.groups, M.n_groups, M.queues);
    return cudaGetLastError();
}

cudaError_t IRT_MARCH_FN(irt_launch_march_batched)(const MarchBatch& M, cudaStream_t st) {
    using namespace IRT_MARCH_NS;
    if (M.n_groups == 0) return cudaSuccess;
    const uint32_t smem = kGroupVec4 * 16 + M.max_scene_bytes;
    typedef decltype(&march_batched_kernel<kAnySampler>) Kernel;
    static const Kernel kernels[] = {march_batched_kernel<kPointF32>, march_batched_kernel<kPointF16>,
                                     march_batched_kernel<kLinearF32>, march_batched_kernel<kAnySampler>};
    if (M.sampler < 0 || M.sampler > kAnySampler) return cudaErrorInvalidValue;
    static KernelFit set_up, march[4];
    int set_up_per_sm, march_per_sm;
    cudaError_t e = set_up.set((const void*)ray_setup_batched_kernel, kSetupThreads, smem, 2, set_up_per_sm);
    const int threads = march_threads(M.sampler);
    if (e == cudaSuccess)
        e = march[M.sampler].set((const void*)kernels[M.sampler], threads, M.max_scene_bytes, march_ctas(M.sampler),
                                 march_per_sm);
    if (e != cudaSuccess) return e;
    const int bps = M.blocks_per_sm > 0 && M.blocks_per_sm < march_per_sm ? M.blocks_per_sm : march_per_sm;
    ray_setup_batched_kernel<<<M.num_sms * set_up_per_sm, kSetupThreads, smem, st>>>(M.groups, M.n_groups, M.queues);
    for (uint32_t g = 0; g < M.n_groups; g += kMarchGroups) {
        MarchGroups part;
        part.n = std::min(M.n_groups - g, kMarchGroups);
        std::copy_n(M.host_groups + g, part.n, part.g);
        kernels[M.sampler]<<<M.num_sms * bps, threads, M.max_scene_bytes, st>>>(part, M.queues);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

#if !IRT_MARCH_FAST
cudaError_t irt_launch_ray_pools_fast(const MarchLaunch& M, cudaStream_t st);
cudaError_t irt_launch_march_fast(const MarchLaunch& M, cudaStream_t st);
cudaError_t irt_launch_ray_pools_batched_fast(const MarchBatch& M, cudaStream_t st);
cudaError_t irt_launch_march_batched_fast(const MarchBatch& M, cudaStream_t st);

cudaError_t irt_launch_ray_pools(const MarchLaunch& M, cudaStream_t st) {
    return M.fast ? irt_launch_ray_pools_fast(M, st) : irt_launch_ray_pools_exact(M, st);
}
cudaError_t irt_launch_march(const MarchLaunch& M, cudaStream_t st) {
    return M.fast ? irt_launch_march_fast(M, st) : irt_launch_march_exact(M, st);
}
cudaError_t irt_launch_ray_pools_batched(const MarchBatch& M, cudaStream_t st) {
    return M.fast ? irt_launch_ray_pools_batched_fast(M, st) : irt_launch_ray_pools_batched_exact(M, st);
}
cudaError_t irt_launch_march_batched(const MarchBatch& M, cudaStream_t st) {
    return M.fast ? irt_launch_march_batched_fast(M, st) : irt_launch_march_batched_exact(M, st);
}

uint32_t irt_march_scene_bytes(uint32_t object_count) {
    return object_count * (uint32_t)sizeof(irtd::MObj);
}
#endif
