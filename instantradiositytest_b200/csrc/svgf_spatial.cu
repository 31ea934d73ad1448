// svgf_spatial.cu — svgf_variance (svgf.wgsl:77-89) and svgf_atrous
// (svgf.wgsl:90-110) as sm_100a CUDA, built with fast math (approximate
// exp, division and square root): these passes only weight and average
// radiance, and their inputs (positions, history length) come exactly from
// the guide and temporal kernels.  Variance in 32x8 blocks, a-trous one thread
// per pixel in blocks of 256 pixels of a row; neighbour taps read through L1.
#include <cuda_runtime.h>

#include "dev_svgf.cuh"
#include "kernels.h"

namespace irtd {

// What a tap reads of a pixel besides its radiance or moments: position (w < 0:
// background), normal and roughness, colour and metal.
struct TapGeometry {
    float4 position, normal, color;
};
// The planes of a row of pixels, from which a tap at a constant distance is
// an immediate offset.  Ld: settled, or written by the kernel before this one
// (the variance pass of a filter that has no temporal one before it).
template <class G, class Ld>
struct TapRow {
    const float4* guide;
    const float4* feat;
    __device__ __forceinline__ TapRow(const SvgfCtx<G>& c, ptrdiff_t i) : guide(c.guide + i), feat(c.feat + 2 * i) {}
    __device__ __forceinline__ TapGeometry at(int32_t dx) const {
        TapGeometry t;
        t.position = Ld::load(guide + dx);
        if constexpr (std::is_same<Ld, Written>::value) {
            asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                         : "=f"(t.normal.x), "=f"(t.normal.y), "=f"(t.normal.z), "=f"(t.normal.w), "=f"(t.color.x),
                           "=f"(t.color.y), "=f"(t.color.z), "=f"(t.color.w)
                         : "l"(feat + 2 * dx)
                         : "memory");
            return t;
        }
        asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
            : "=f"(t.normal.x), "=f"(t.normal.y), "=f"(t.normal.z), "=f"(t.normal.w), "=f"(t.color.x),
              "=f"(t.color.y), "=f"(t.color.z), "=f"(t.color.w)
            : "l"(feat + 2 * dx));
        return t;
    }
};

// A pixel's own terms of the geometry weight of its taps (svgf.wgsl:32-44).
struct TapCentre {
    V3 position, normal, color;
    float rough, metal;
    float kz;  // log2(e) over the plane-distance tolerance
    __device__ __forceinline__ void set(const TapGeometry& own, float step) {
        position = xyz(own.position);
        normal = xyz(own.normal);
        color = xyz(own.color);
        rough = own.normal.w;
        metal = own.color.w;
        kz = 1.44269504f / wmax(.0001f, own.position.w * (step * .5f));
    }
    // The tap's normal weight, and in `geom` the plane-distance, colour and
    // parameter terms as one exponent of 2; false where the weight is 0
    // (background, or one of its factors underflows).
    __device__ __forceinline__ bool weigh(const TapGeometry& t, float& wn, float& geom) const {
        const float kc = 8.f * 1.44269504f;
        wn = pow64(wmax(dot(normal, xyz(t.normal)), 0.f));
        const V3 dc = color - xyz(t.color);
        const float d0 = rough - t.normal.w, d1 = metal - t.color.w;
        geom = fmaf(length(dc) + sqrtf(fmaf(d0, d0, d1 * d1)), kc, fabsf(dot(xyz(t.position) - position, normal)) * kz);
        return !(t.position.w < 0.f || !(wn > 0.f) || geom > 126.f);
    }
};

// svgf.wgsl:77-89
// With MomF16 (mean, deviation) moments the 7x7 sums are taken about the
// centre pixel's mean (shifted data), so E[l^2] - E[l]^2 is formed from
// small numbers: s0 = sum w (m - K), s1 = sum w (dev^2 + (m - K)^2).
// The sums of svgf_variance over the taps of one pixel.
template <class M>
struct VarianceSums {
    float s0 = 0.f, s1 = 0.f, total = 0.f;
    // The row of taps py + yy; without a branch before the sums, so that its
    // seven taps' loads issue together.
    template <class G>
    __device__ __forceinline__ void row(const SvgfCtx<G>& c, const TapCentre& a, const typename M::T* moments, float K,
                                        int32_t W, int32_t H, int32_t px, int32_t py, int32_t yy) {
        const int32_t qy = py + yy;
        const bool row_in = yy <= 3 && qy >= 0 && qy < H;
        const ptrdiff_t at = (ptrdiff_t)min(max(qy, 0), H - 1) * W;
#pragma unroll
        for (int32_t xx = -3; xx <= 3; xx++) {
            const int32_t qx = px + xx;
            const ptrdiff_t q = at + min(max(qx, 0), W - 1);
            const TapGeometry g = TapRow<G, Written>(c, q).at(0);
            const Moments m = M::load(moments, q);
            float wn, geom;
            const bool counts = a.weigh(g, wn, geom) && row_in && qx >= 0 && qx < W;
            const float w = wn * exp2f(-geom);
            if (!counts) continue;
            if constexpr (M::central) {
                float d = m.mean - K;
                s0 += d * w;
                s1 += fmaf(m.second, m.second, d * d) * w;
            } else {
                s0 += m.mean * w;
                s1 += m.second * w;
            }
            total += w;
        }
    }
    __device__ __forceinline__ void add(const VarianceSums& o) {
        s0 += o.s0;
        s1 += o.s1;
        total += o.total;
    }
    __device__ __forceinline__ float sigma(float age) const {
        const float dn = wmax(total, .00001f);
        const float m0 = s0 / dn, m1 = s1 / dn;
        return sqrtf(wmax(m1 - m0 * m0, 0.f) * 4.f / wmax(age, 1.f));
    }
};

// Only pixels with a young history (disocclusions; every pixel of the first
// frames) take the 49 taps.  A block of 256 lists its young pixels.  Up to 64
// of them: eight lanes take a pixel, a row of taps each, since what a few
// young pixels cost is the latency of their loads one after the other.  More:
// a thread a pixel, whose loads coalesce.  160x100 25 -> 12 us, 480x300 31 -> 18,
// 960x600 with moving objects 44 -> 32, 1920x1200 f32 / mixed 96 / 101 -> 82 / 76;
// all young at 1920x1200 355 -> 312 (1235 with eight lanes each).  Lists up to
// 32 leave 160x100 at 14, up to 128 take 960x600 to 43.
constexpr uint32_t kSpreadYoung = 64;
template <class G, class R, class M>
__device__ __forceinline__ void variance_body(const irt_frame& f, const SvgfCtx<G>& c, const typename R::T* input,
                                              const typename M::T* moments, typename R::T* out, int32_t x, int32_t y) {
    __shared__ int2 list[256];  // whole coordinates: frames may be wider than 16 bits hold
    __shared__ uint32_t listed;
    const unsigned full = 0xffffffffu;
    const int32_t W = (int32_t)f.size[0], H = (int32_t)f.size[1];
    const uint32_t t = threadIdx.y * blockDim.x + threadIdx.x, lane = t & 31u;
    if (t == 0) listed = 0u;
    __syncthreads();
    bool young = false;
    if (x < W && y < H) {
        const ptrdiff_t i = (ptrdiff_t)y * W + x;
        young = M::load(moments, i).age < 4.f && !(load_written(&c.guide[i].w) < 0.f);  // depth < 1
        if (!young) {
            float4 in = R::load(input, i);
            in.w = wmin(in.w, 65000.f);
            R::store(out, i, in);
        }
    }
    const unsigned in_warp = __ballot_sync(full, young);
    uint32_t base = 0;
    if (lane == 0u && in_warp) base = atomicAdd(&listed, (uint32_t)__popc(in_warp));
    base = __shfl_sync(full, base, 0);
    if (young) list[base + (uint32_t)__popc(in_warp & ((1u << lane) - 1u))] = make_int2(x, y);
    __syncthreads();
    const uint32_t n = listed;
    auto pixel = [&](uint32_t k, auto&& sums) {
        const int32_t px = list[k].x, py = list[k].y;
        const ptrdiff_t i = (ptrdiff_t)py * W + px;
        const Moments centre = M::load(moments, i);
        TapCentre a;
        a.set(TapRow<G, Written>(c, i).at(0), 1.f);
        VarianceSums<M> v;
        if (!sums(v, a, M::central ? centre.mean : 0.f, px, py)) return;
        const float4 in = R::load(input, i);
        R::store(out, i, make_float4(in.x, in.y, in.z, wmin(v.sigma(centre.age), 65000.f)));
    };
    if (n > kSpreadYoung) {
        if (t < n)
            pixel(t, [&](VarianceSums<M>& v, const TapCentre& a, float K, int32_t px, int32_t py) {
                // rows added as the eight lanes' exchange adds them, so that a
                // pixel's value does not depend on its block's list
                VarianceSums<M> hold, half;
#pragma unroll 1
                for (int32_t k = 0; k < 7; k++) {
                    VarianceSums<M> r;
                    r.row(c, a, moments, K, W, H, px, py, k - 3);
                    if ((k & 1) == 0) {
                        hold = r;
                        continue;
                    }
                    hold.add(r);
                    if (k == 1) v = hold;
                    if (k == 3) v.add(hold);
                    if (k == 5) half = hold;
                }
                half.add(hold);
                v.add(half);
                return true;
            });
        return;
    }
    for (uint32_t k = t / 8u; k - lane / 8u < n; k += blockDim.x * blockDim.y / 8u)  // whole warps
        pixel(min(k, n - 1u), [&](VarianceSums<M>& v, const TapCentre& a, float K, int32_t px, int32_t py) {
            v.row(c, a, moments, K, W, H, px, py, (int32_t)(lane & 7u) - 3);
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                v.s0 += __shfl_xor_sync(full, v.s0, o);
                v.s1 += __shfl_xor_sync(full, v.s1, o);
                v.total += __shfl_xor_sync(full, v.total, o);
            }
            return k < n && (lane & 7u) == 0u;
        });
}

template <class G, class R, class M>
__global__ void __launch_bounds__(256, 4) svgf_variance_kernel(const __grid_constant__ irt_frame f, const __grid_constant__ SvgfCtx<G> c,
                                                            const typename R::T* input, const typename M::T* moments,
                                                            typename R::T* out) {
    frame_kernel_begin();
    variance_body<G, R, M>(f, c, input, moments, out, blockIdx.x * blockDim.x + threadIdx.x,
                           blockIdx.y * blockDim.y + threadIdx.y);
}

// A-trous: 25 taps a pixel, bound by L1 bandwidth (64 bytes a tap with f32
// radiance) and load latency.  Per 1920x1200 pass, f32 / mixed storage, 256 / 246 us
// before: a tap reads the guide and the feature record (one 128-bit and one
// 256-bit load, also for f32 planes, whose five loads a tap cost 197 us with
// all of the following), the wavelet step is a template constant so that the
// taps of a row are immediate offsets, interior pixels test no bounds, the
// three exponentials of a tap are one exp2 of the summed exponents with the
// two divisors inverted once a pixel, no branch stands between the loads of
// one tap and the next, and the 25 taps are unrolled (179 / 166 us with the
// rows rolled): 173 / 156 us.  Two pixels a step apart per thread (30 taps
// read instead of 50) 182 / 180; blocks of 32x4 176 us for step 1, 194-215 for
// the others.
//
constexpr __device__ __host__ float wavelet_kernel(int32_t x) {
    return x == 0 ? 1.f : (x == 1 || x == -1) ? 2.f / 3.f : 1.f / 6.f;
}

// One pixel of svgf_atrous with its sums.
struct Atrous {
    TapCentre c;
    float lum, kl;  // log2(e) over phi
    V3 sum;
    float total, v;
    // svgf.wgsl:99-105: the exponentials of the geometry and luminance terms
    // as one exp2 of their sum, the divisors' reciprocals taken once a pixel.
    // Without a branch before the sums, so that the loads of later taps issue
    // ahead of this one's arithmetic.
    __device__ __forceinline__ void tap(const TapGeometry& t, float4 smp, float kernel) {
        float wn, geom;
        const bool counts = c.weigh(t, wn, geom);
        const float w = wn * kernel * exp2f(-(geom + fabsf(luminance(xyz(smp)) - lum) * kl));
        if (!counts) return;
        sum = sum + xyz(smp) * w;
        v += smp.w * smp.w * w * w;
        total += w;
    }
};

// The pixel's own terms; false: background, whose radiance passes through.
template <class G, class R>
__device__ __forceinline__ bool atrous_begin(Atrous& a, const SvgfCtx<G>& c, const typename R::T* input,
                                             typename R::T* out, typename R::T* out2, int32_t W, int32_t H,
                                             int32_t x, int32_t y, float step) {
    const ptrdiff_t i = (ptrdiff_t)y * W + x;
    const float4 c4 = R::load(input, i);
    const TapGeometry own = TapRow<G, Settled>(c, i).at(0);
    if (own.position.w < 0.f) {  // depth >= 1
        R::store(out, i, c4);
        if (out2) R::store(out2, i, c4);
        return false;
    }
    float variance = 0.f;
#pragma unroll
    for (int32_t yy = -1; yy <= 1; yy++) {
        const int32_t qy = min(max(y + yy, 0), H - 1);
#pragma unroll
        for (int32_t xx = -1; xx <= 1; xx++) {
            const int32_t qx = min(max(x + xx, 0), W - 1);
            const float s = R::load(input, (size_t)qy * W + qx).w;
            variance += s * s * ((xx == 0 ? 2.f : 1.f) * (yy == 0 ? 2.f : 1.f));
        }
    }
    a.c.set(own, step);
    a.lum = luminance(xyz(c4));
    a.kl = 1.44269504f / (4.f * sqrtf(variance * (1.f / 16.f)) + .0001f);
    a.sum = V3{0.f, 0.f, 0.f};
    a.total = a.v = 0.f;
    return true;
}
template <class R>
__device__ __forceinline__ void atrous_end(const Atrous& a, typename R::T* out, typename R::T* out2, ptrdiff_t i) {
    const float dn = 1.f / wmax(a.total, .00001f);
    const float4 o = make_float4(a.sum.x * dn, a.sum.y * dn, a.sum.z * dn, wmin(sqrtf(a.v) * dn, 65000.f));
    R::store(out, i, o);
    if (out2) R::store(out2, i, o);
}

// svgf.wgsl:91-110 with the wavelet's step as a constant; `out2` (optional)
// receives a second copy of the result.
template <class G, class R, int32_t Step>
__device__ __forceinline__ void atrous_body(const irt_frame& f, const SvgfCtx<G>& c, const typename R::T* input,
                                            typename R::T* out, typename R::T* out2, int32_t x, int32_t y) {
    const int32_t W = (int32_t)f.size[0], H = (int32_t)f.size[1];
    if (x >= W || y >= H) return;
    const ptrdiff_t i = (ptrdiff_t)y * W + x;
    Atrous a;
    if (!atrous_begin<G, R>(a, c, input, out, out2, W, H, x, y, (float)Step)) return;
    if (x >= 2 * Step && y >= 2 * Step && x < W - 2 * Step && y < H - 2 * Step) {
#pragma unroll
        for (int32_t yy = -2; yy <= 2; yy++) {
            const TapRow<G, Settled> row(c, i + (ptrdiff_t)(yy * Step) * W);
            const typename R::T* in = input + i + (ptrdiff_t)(yy * Step) * W;
#pragma unroll
            for (int32_t xx = -2; xx <= 2; xx++)
                a.tap(row.at(xx * Step), R::load(in, xx * Step), wavelet_kernel(xx) * wavelet_kernel(yy));
        }
    } else {
#pragma unroll 1
        for (int32_t k = 0; k < 25; k++) {
            const int32_t xx = k % 5 - 2, yy = k / 5 - 2, qx = x + xx * Step, qy = y + yy * Step;
            if (qx < 0 || qy < 0 || qx >= W || qy >= H) continue;
            const ptrdiff_t q = (ptrdiff_t)qy * W + qx;
            a.tap(TapRow<G, Settled>(c, q).at(0), R::load(input, q), wavelet_kernel(xx) * wavelet_kernel(yy));
        }
    }
    atrous_end<R>(a, out, out2, i);
}

template <class G, class R, int32_t Step>
__global__ void __launch_bounds__(256, 4) svgf_atrous_kernel(const __grid_constant__ irt_frame f, const __grid_constant__ SvgfCtx<G> c,
                                                          const typename R::T* input, typename R::T* __restrict__ out, typename R::T* __restrict__ out2) {
    frame_kernel_begin();
    atrous_body<G, R, Step>(f, c, input, out, out2, blockIdx.x * blockDim.x + threadIdx.x,
                            blockIdx.y * blockDim.y + threadIdx.y);
}

// Calls fn(integral_constant) for a wavelet step 1, 2, 4, 8 or 16 (at most 5 iterations).
template <class Fn>
static cudaError_t with_step(int step, Fn&& fn) {
    switch (step) {
    case 1: return fn(std::integral_constant<int32_t, 1>{});
    case 2: return fn(std::integral_constant<int32_t, 2>{});
    case 4: return fn(std::integral_constant<int32_t, 4>{});
    case 8: return fn(std::integral_constant<int32_t, 8>{});
    case 16: return fn(std::integral_constant<int32_t, 16>{});
    }
    return cudaErrorInvalidValue;
}

template <class G, class R, class M>
__global__ void __launch_bounds__(256, 4) svgf_variance_batched(const irt_frame* __restrict__ frames,
                                                             const SView<G>* __restrict__ views,
                                                             const uint32_t* __restrict__ tile_start, uint32_t n) {
    const uint32_t v = svgf_find_view(tile_start, n, blockIdx.x);
    __shared__ __align__(16) irt_frame f;
    __shared__ __align__(16) SView<G> w;
    svgf_stage(frames + v, &f);
    svgf_stage(views + v, &w);
    __syncthreads();
    int32_t x, y;
    svgf_tile_xy(f.size[0], blockIdx.x - __ldg(tile_start + v), x, y);
    typedef typename R::T T;
    variance_body<G, R, M>(f, w.c, (const T*)w.in, (const typename M::T*)w.moments_in, (T*)w.out, x, y);
}

template <class G, class R, int32_t Step>
__global__ void __launch_bounds__(256, 4) svgf_atrous_batched(const irt_frame* __restrict__ frames,
                                                           const SView<G>* __restrict__ views,
                                                           const uint32_t* __restrict__ tile_start, uint32_t n) {
    const uint32_t v = svgf_find_view(tile_start, n, blockIdx.x);
    __shared__ __align__(16) irt_frame f;
    __shared__ __align__(16) SView<G> w;
    svgf_stage(frames + v, &f);
    svgf_stage(views + v, &w);
    __syncthreads();
    int32_t x, y;
    svgf_tile_xy(f.size[0], blockIdx.x - __ldg(tile_start + v), x, y);
    typedef typename R::T T;
    atrous_body<G, R, Step>(f, w.c, (const T*)w.in, (T*)w.out, (T*)w.out2, x, y);
}

template <class G, class R, class M>
static cudaError_t spatial_typed(const SvgfLaunch& L, int stage, cudaStream_t st) {
    SvgfCtx<G> c = make_ctx<G>(L);
    const irt_frame& f = *L.frame;
    typedef typename R::T T;
    if (stage == 1) {
        dim3 block(32, 8);
        dim3 grid((f.size[0] + 31) / 32, (f.size[1] + 7) / 8);
        return launch_behind(svgf_variance_kernel<G, R, M>, grid, block, 0, st, f, c, (const T*)L.in,
                             (const typename M::T*)L.moments_in, (T*)L.out);
    }
    if (stage == 2) {
        // Blocks of 256 pixels of one row (4 passes at 1920x1200 f32: 0.72 ms; 64x2 0.77, 32x4
        // 0.77).
        dim3 block(256, 1);
        dim3 grid((f.size[0] + 255) / 256, f.size[1]);
        return with_step(L.step, [&](auto step) {
            return launch_behind(svgf_atrous_kernel<G, R, decltype(step)::value>, grid, block, 0, st, f, c,
                                 (const T*)L.in, (T*)L.out, (T*)L.out2);
        });
    }
    return cudaErrorInvalidValue;
}

template <class G, class R, class M>
static cudaError_t spatial_batched_typed(const BatchLaunch& B, int stage, cudaStream_t st) {
    const SView<G>* views = static_cast<const SView<G>*>(B.table);
    dim3 block(B.bx, B.by);
    if (stage == 1)
        svgf_variance_batched<G, R, M><<<B.tiles, block, 0, st>>>(B.frames, views, B.tile_start, B.n);
    else if (stage == 2)
        return with_step(B.step, [&](auto step) {
            svgf_atrous_batched<G, R, decltype(step)::value><<<B.tiles, block, 0, st>>>(B.frames, views, B.tile_start,
                                                                                       B.n);
            return cudaGetLastError();
        });
    else
        return cudaErrorInvalidValue;
    return cudaGetLastError();
}

}  // namespace irtd

cudaError_t irt_launch_svgf_spatial_batched(const BatchLaunch& B, int stage, cudaStream_t st) {
    using namespace irtd;
    SvgfLaunch L{};
    L.gbuffer.format = B.gbuffer_format;
    L.radiance_f16 = B.radiance_f16;
    L.moments_f16 = stage == 2 ? 0 : B.moments_f16;
    return dispatch_svgf(L, [&](auto g, auto r, auto m) {
        return spatial_batched_typed<decltype(g), decltype(r), decltype(m)>(B, stage, st);
    });
}

cudaError_t irt_launch_svgf_spatial(const SvgfLaunch& L, int stage, cudaStream_t st) {
    using namespace irtd;
    if (stage == 2) {  // a-trous reads no moments
        SvgfLaunch A = L;
        A.moments_f16 = 0;
        return dispatch_svgf(A, [&](auto g, auto r, auto) {
            return spatial_typed<decltype(g), decltype(r), MomF32>(A, stage, st);
        });
    }
    return dispatch_svgf(L, [&](auto g, auto r, auto m) {
        return spatial_typed<decltype(g), decltype(r), decltype(m)>(L, stage, st);
    });
}
