// trace_plain.cu - the plain form: megakernels that reproduce the reference's
// compute-only shader (shaders/ray_trace.comp.hybrid.hlsl) operation for
// operation, one thread per ray or per pixel.  This is the parity baseline the
// optimised kernels are measured against.
#include "exact_trace.cuh"
#include "kernels.h"
#include "shade.cuh"
#include "trace_common.cuh"

namespace ae {

// ---------------------------------------------------------------------------
// Closest hit over a ray batch
// ---------------------------------------------------------------------------
// WT: the watertight triangle test in the same walk (AE_VARIANT_PLAIN_WT).
template <bool WT>
__global__ void __launch_bounds__(128) k_closest_plain(DevScene S, const ae_ray *__restrict__ rays, uint32_t n,
                                                       ae_hit *__restrict__ hits) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 *rp = reinterpret_cast<const float4 *>(rays + i);
    const float4 r0 = __ldg(rp), r1 = __ldg(rp + 1);
    uint32_t seed = 1u;
    DHit h;
    ae_hit out;
    out.t = 0.0f; out.alpha = 0.0f; out.beta = 0.0f; out.object = AE_MISS; out.prim = AE_MISS;
    if (traverse_ref<WT>(S, mk(r0.x, r0.y, r0.z), mk(r1.x, r1.y, r1.z), r1.w, r0.w, h, seed)) {
        out.t = h.t; out.alpha = h.alpha; out.beta = h.beta; out.object = h.slot; out.prim = h.prim;
    }
    hits[i] = out;
}

// The debug walk (AE_VARIANT_PLAIN_CHECKED): PLAIN's traversal with every
// stack push and buffer index checked (Checks).
__global__ void __launch_bounds__(128) k_closest_checked(DevScene S, Checks C, const ae_ray *__restrict__ rays,
                                                         uint32_t n, ae_hit *__restrict__ hits) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 *rp = reinterpret_cast<const float4 *>(rays + i);
    const float4 r0 = __ldg(rp), r1 = __ldg(rp + 1);
    uint32_t seed = 1u;
    DHit h;
    ae_hit out;
    out.t = 0.0f; out.alpha = 0.0f; out.beta = 0.0f; out.object = AE_MISS; out.prim = AE_MISS;
    if (traverse_ref<false>(S, mk(r0.x, r0.y, r0.z), mk(r1.x, r1.y, r1.z), r1.w, r0.w, h, seed, nullptr, &C)) {
        out.t = h.t; out.alpha = h.alpha; out.beta = h.beta; out.object = h.slot; out.prim = h.prim;
    }
    hits[i] = out;
}

cudaError_t launch_closest_checked(const DevScene &S, const Checks &C, const ae_ray *rays, uint32_t n, ae_hit *hits,
                                   cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    k_closest_checked<<<(n + 127) / 128, 128, 0, st>>>(S, C, rays, n, hits);
    return cudaGetLastError();
}

// The same traversal with its touches counted: the algorithmic traffic of
// the reference's walk, per ray set, summed in 64-bit.
__global__ void __launch_bounds__(128) k_count_plain(DevScene S, const ae_ray *__restrict__ rays, uint32_t n,
                                                     unsigned long long *__restrict__ totals) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    Touch T = {0, 0, 0, 0, 0, 0, 0};
    if (i < n) {
        const float4 *rp = reinterpret_cast<const float4 *>(rays + i);
        const float4 r0 = __ldg(rp), r1 = __ldg(rp + 1);
        uint32_t seed = 1u;
        DHit h;
        traverse_ref(S, mk(r0.x, r0.y, r0.z), mk(r1.x, r1.y, r1.z), r1.w, r0.w, h, seed, &T);
    }
    const uint32_t v[6] = {T.tlas, T.objects, T.instances, T.blas, T.tris, T.winners};
    for (int k = 0; k < 6; k++) {
        unsigned long long x = v[k];
        for (int off = 16; off > 0; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
        if ((threadIdx.x & 31) == 0 && x) atomicAdd(totals + k, x);
    }
}

// ---------------------------------------------------------------------------
// Compute-only path tracer (hybrid:1230-1404)
// ---------------------------------------------------------------------------
// CalculateDirectLight, hybrid:1122-1212.
// T (optional): touch counters of the shadow traversals.
AE_DEV f3 direct_light(const DevScene &S, const DHit &h, f3 surf_albedo, float time, uint32_t &seed,
                       Touch *T = nullptr) {
    f3 acc = splat(0.0f);
    for (uint32_t i = 0; i < S.n_lights; i++) {
        const ae_object *L = S.objects + __ldg(S.lights + i);
        const ObjHead lh = load_head(L);
        f3 lp;
        float omega;
        sample_light(L, lh.shape, h.p, lp, omega, seed);
        if (omega <= 0.0f) continue;
        f3 sd = lp - h.p;
        const float dist = length(sd);
        if (dist <= 1e-6f) continue;
        sd = sd / dist;
        const float ct = dot(h.n, sd);
        if (ct <= 0.0f) continue;
        f3 so = h.p + h.n * 0.001f;
        bool occluded = false;
        for (int k = 0; k < 4; k++) {
            DHit sh;
            if (!traverse_ref(S, so, sd, time, 0.001f, sh, seed, T)) break;
            if (sh.t >= AE_SUB(distance(lp, so), 0.001f)) break;
            const uint32_t mt = load_head(S.objects + sh.slot).material;
            if (mt == AE_MAT_DIFFUSE_LIGHT) break;
            if (mt != AE_MAT_DIELECTRIC) { occluded = true; break; }
            so = sh.p + sd * 0.001f;
        }
        if (!occluded) {
            const MatRec lm = load_mat(L);
            const f3 rad = lm.emission * lm.albedo;
            acc = acc + surf_albedo * rad * ct * omega;
        }
    }
    return acc;
}

// ColorRay, hybrid:1230-1325.  T (optional) counts every traversal's touches.
AE_DEV f3 color_ray(const DevScene &S, const FrameParams &F, f3 o, f3 d, float time, uint32_t &seed,
                    Touch *T = nullptr) {
    f3 thr = splat(1.0f), acc = splat(0.0f);
    for (uint32_t b = 0; b < F.depth; b++) {
        DHit h;
        if (!traverse_ref(S, o, d, time, 0.001f, h, seed, T)) {
            acc = acc + thr * F.sky;
            break;
        }
        const MatRec m = load_mat(S.objects + h.slot);
        if (m.type == AE_MAT_DIFFUSE_LIGHT) {
            acc = acc + thr * (m.emission * m.albedo);
            break;
        }
        // SurfaceAlbedo (textured when the material has a layer).
        const f3 alb = m.type != AE_MAT_DIELECTRIC ? surface_albedo(S, h, m, o, d) : m.albedo;
        if (m.type == AE_MAT_LAMBERTIAN) {
            f3 dl = direct_light(S, h, alb, time, seed, T);
            const float luma = maxc(dl);
            if (luma > 8.0f) dl = dl * AE_DIV(8.0f, luma);
            acc = acc + thr * dl;
        }
        f3 sd, gw;
        if (!get_bounce(d, h, m, alb, sd, gw, seed)) break;
        d = normalize(sd);
        const float sgn = dot(d, h.n) < 0.0f ? -1.0f : 1.0f;
        o = h.p + h.n * AE_MUL(0.001f, sgn);
        if (m.type == AE_MAT_GGX_METAL) thr = thr * gw;
        else if (m.type != AE_MAT_DIELECTRIC) thr = thr * alb;
        if (b > 0) {
            const float p = clampf(maxc(thr), 0.1f, 1.0f);
            if (rng_next(seed) > p) break;
            thr = thr / p;
        }
    }
    return acc;
}

// The reference walk for the rays that the exact walk leaves undecided.
__device__ __noinline__ bool traverse_undecided(const DevScene &S, f3 o, f3 d, float time, float tn, DHit &h,
                                                uint32_t &seed) {
    return traverse_ref(S, o, d, time, tn, h, seed);
}

// The same on the optimised structures (exact_trace.cuh; the reference walk
// where those leave a ray undecided), as one loop whose turns each trace one
// ray: the path's next segment or one step of a light sample's shadow loop.
// The walk then stands in the code once, and lanes that need no shadow ray
// trace their next segment beside those that do (480x270 frames: 17 objects
// of 160 triangles 365 -> 309 us, 66 of 59,398 674 -> 580 us against two
// inlined walks).  Random numbers are drawn in the reference's order.
AE_DEV f3 color_ray_exact(const DevScene &S, const ExactView &X, const FrameParams &F, f3 o, f3 d, float time,
                          uint32_t &seed, uint2 *stk) {
    f3 thr = splat(1.0f), acc = splat(0.0f);
    if (F.depth == 0) return acc;
    DHit h;
    f3 din = d, alb, dl, c, lp;  // the segment's direction, the surface's albedo, light sum, sample, light point
    uint32_t b = 0, light = 0;
    int step = 0;
    bool shadow = false;
    for (;;) {
        const float lim = shadow ? AE_SUB(distance(lp, o), 0.001f) : kFarStart;
        // The hit's surface goes to h on a path segment; a shadow ray needs its
        // distance and object alone.
        bool hit;
        float t = 0.0f;
        uint32_t slot = 0;
        Best w;
        const int v = closest_exact<kAllObjects, kSharedStack>(S, X, o, d, time, 0.001f, lim, kFarStart, w, stk,
                                                               threadIdx.x, 128);
        if (v == kUndecided) {
            DHit r;
            hit = traverse_undecided(S, o, d, time, 0.001f, r, seed);
            if (hit) {
                t = r.t;
                slot = r.slot;
                if (!shadow) h = r;
            }
        } else {
            hit = v == kExactHit;
            if (hit) {
                t = w.t;
                slot = w.object;
                if (!shadow) exact_hit_record(S, w, o, d, time, h);
            }
        }
        bool lights = true;
        if (!shadow) {
            if (!hit) {
                acc = acc + thr * F.sky;
                break;
            }
            const MatRec m = load_mat(S.objects + h.slot);
            if (m.type == AE_MAT_DIFFUSE_LIGHT) {
                acc = acc + thr * (m.emission * m.albedo);
                break;
            }
            // SurfaceAlbedo (textured when the material has a layer).
            alb = m.type != AE_MAT_DIELECTRIC ? surface_albedo(S, h, m, o, d) : m.albedo;
            lights = m.type == AE_MAT_LAMBERTIAN;
            dl = splat(0.0f);
            light = 0;
        } else {
            // The reference's shadow loop: up to four closest hits, stepping
            // through glass; lights and hits past the light point do not block.
            bool occluded = false;
            if (hit && !(t >= lim)) {  // a NaN distance blocks, as the reference's comparison has it
                const uint32_t mt = load_head(S.objects + slot).material;
                occluded = mt != AE_MAT_DIFFUSE_LIGHT && mt != AE_MAT_DIELECTRIC;
                if (mt == AE_MAT_DIELECTRIC && ++step < 4) {
                    o = (o + d * t) + d * 0.001f;
                    continue;
                }
            }
            if (!occluded) dl = dl + c;
            light++;
        }
        if (lights) {
            // The next light sample that needs a shadow ray.
            shadow = false;
            for (; light < S.n_lights; light++) {
                const ae_object *L = S.objects + __ldg(S.lights + light);
                const ObjHead lh = load_head(L);
                float omega;
                sample_light(L, lh.shape, h.p, lp, omega, seed);
                if (omega <= 0.0f) continue;
                f3 sd = lp - h.p;
                const float dist = length(sd);
                if (dist <= 1e-6f) continue;
                sd = sd / dist;
                const float ct = dot(h.n, sd);
                if (ct <= 0.0f) continue;
                const MatRec lm = load_mat(L);
                const f3 rad = lm.emission * lm.albedo;
                c = alb * rad * ct * omega;
                o = h.p + h.n * 0.001f;
                d = sd;
                step = 0;
                shadow = true;
                break;
            }
            if (shadow) continue;
            const float luma = maxc(dl);
            if (luma > 8.0f) dl = dl * AE_DIV(8.0f, luma);
            acc = acc + thr * dl;
        }
        const MatRec m = load_mat(S.objects + h.slot);
        f3 sd, gw;
        if (!get_bounce(din, h, m, alb, sd, gw, seed)) break;
        d = normalize(sd);
        const float sgn = dot(d, h.n) < 0.0f ? -1.0f : 1.0f;
        o = h.p + h.n * AE_MUL(0.001f, sgn);
        if (m.type == AE_MAT_GGX_METAL) thr = thr * gw;
        else if (m.type != AE_MAT_DIELECTRIC) thr = thr * alb;
        if (b > 0) {
            const float p = clampf(maxc(thr), 0.1f, 1.0f);
            if (rng_next(seed) > p) break;
            thr = thr / p;
        }
        din = d;
        if (++b >= F.depth) break;
    }
    return acc;
}

// main, hybrid:1328-1404.  Threads cover 16x8 pixel tiles so a warp's rays
// start coherent; the result per pixel does not depend on the mapping.  A warp
// takes 16x2 pixels on the exact walk and 8x4 on the reference walk, which
// scenes with media use (480x270 frames of 66 objects: 580 against 658 us on
// the exact walk; the Cornell box 376 -> 365 us on the reference walk).
template <bool EXACT>
__global__ void __launch_bounds__(128) k_render_plain(DevScene S, ExactView X, FrameParams F, float4 *__restrict__ accum,
                                                      uchar4 *__restrict__ display, float4 *__restrict__ frame) {
    extern __shared__ uint2 stk[];
    const uint32_t t = threadIdx.x;
    const uint32_t x = blockIdx.x * 16 + (EXACT ? (t & 15) : (t >> 5 & 1) * 8 + (t & 7));
    const uint32_t y = blockIdx.y * 8 + (EXACT ? t >> 4 : (t >> 6) * 4 + (t >> 3 & 3));
    if (x >= F.width || y >= F.height) return;
    const size_t px = size_t(y) * F.width + x;
    if (F.display_only) {
        const float4 a = accum[px];
        display[px] = display_texel(mk(a.x, a.y, a.z), F.exposure);
        return;
    }
    uint32_t seed = x + y * F.width + F.batch * F.width * F.height + 1u;
    f3 color = splat(0.0f);
    for (uint32_t s = 0; s < F.spp; s++) {
        const float jx = AE_SUB(rng_next(seed), 0.5f);
        const float jy = AE_SUB(rng_next(seed), 0.5f);
        const f3 tgt = F.pixel0 + AE_ADD(AE_U2F(x), jx) * F.pixel_u + AE_ADD(AE_U2F(y), jy) * F.pixel_v;
        f3 o = F.source;
        if (F.defocus_angle > 0.0f) {
            float px_, py_;
            for (;;) {
                const float a = rng_next(seed), b = rng_next(seed);
                px_ = AE_SUB(AE_MUL(a, 2.0f), 1.0f);
                py_ = AE_SUB(AE_MUL(b, 2.0f), 1.0f);
                if (length(mk(px_, py_, 0.0f)) < 1.0f) break;
            }
            o = F.source + px_ * F.defocus_u + py_ * F.defocus_v;
        }
        const f3 d = normalize(tgt - o);
        const float time = rng_next(seed);
        color = color + (EXACT ? color_ray_exact(S, X, F, o, d, time, seed, stk) : color_ray(S, F, o, d, time, seed));
    }
    color = color / AE_U2F(F.spp);
    if (frame) frame[px] = make_float4(color.x, color.y, color.z, 1.0f);
    f3 acc;
    if (F.batch == 0) {
        acc = color;
    } else {
        const float4 prev = accum[px];
        const float w = AE_DIV(1.0f, AE_U2F(F.batch + 1));
        acc = lerp(mk(prev.x, prev.y, prev.z), color, w);
    }
    accum[px] = make_float4(acc.x, acc.y, acc.z, 1.0f);
    display[px] = display_texel(acc, F.exposure);
}

// The frame's paths (main's camera ray and ColorRay, spp samples per pixel)
// with every traversal's touches counted - the algorithmic traffic per path
// of the reference's megakernel.  Writes no image; outside timed regions.
__global__ void __launch_bounds__(128) k_count_paths(DevScene S, FrameParams F,
                                                     unsigned long long *__restrict__ totals) {
    const uint32_t x = blockIdx.x * 16 + (threadIdx.x & 15);
    const uint32_t y = blockIdx.y * 8 + (threadIdx.x >> 4);
    Touch T = {0, 0, 0, 0, 0, 0, 0};
    if (x < F.width && y < F.height) {
        uint32_t seed = x + y * F.width + F.batch * F.width * F.height + 1u;
        for (uint32_t s = 0; s < F.spp; s++) {
            const float jx = AE_SUB(rng_next(seed), 0.5f);
            const float jy = AE_SUB(rng_next(seed), 0.5f);
            const f3 tgt = F.pixel0 + AE_ADD(AE_U2F(x), jx) * F.pixel_u + AE_ADD(AE_U2F(y), jy) * F.pixel_v;
            f3 o = F.source;
            if (F.defocus_angle > 0.0f) {
                float px_, py_;
                for (;;) {
                    const float a = rng_next(seed), b = rng_next(seed);
                    px_ = AE_SUB(AE_MUL(a, 2.0f), 1.0f);
                    py_ = AE_SUB(AE_MUL(b, 2.0f), 1.0f);
                    if (length(mk(px_, py_, 0.0f)) < 1.0f) break;
                }
                o = F.source + px_ * F.defocus_u + py_ * F.defocus_v;
            }
            const f3 d = normalize(tgt - o);
            const float time = rng_next(seed);
            color_ray(S, F, o, d, time, seed, &T);
        }
    }
    const uint32_t v[7] = {T.tlas, T.objects, T.instances, T.blas, T.tris, T.winners, T.rays};
    for (int k = 0; k < 7; k++) {
        unsigned long long c = v[k];
        for (int off = 16; off > 0; off >>= 1) c += __shfl_down_sync(0xffffffffu, c, off);
        if ((threadIdx.x & 31) == 0 && c) atomicAdd(totals + k, c);
    }
}

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------
cudaError_t launch_closest_plain(const DevScene &S, const ae_ray *rays, uint32_t n, ae_hit *hits, cudaStream_t st,
                                 bool watertight) {
    if (n == 0) return cudaSuccess;
    if (watertight) k_closest_plain<true><<<(n + 127) / 128, 128, 0, st>>>(S, rays, n, hits);
    else k_closest_plain<false><<<(n + 127) / 128, 128, 0, st>>>(S, rays, n, hits);
    return cudaGetLastError();
}

cudaError_t launch_count_plain(const DevScene &S, const ae_ray *rays, uint32_t n, unsigned long long *totals,
                               cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    k_count_plain<<<(n + 127) / 128, 128, 0, st>>>(S, rays, n, totals);
    return cudaGetLastError();
}

cudaError_t launch_count_paths(const DevScene &S, const FrameParams &F, unsigned long long *totals, cudaStream_t st) {
    dim3 grid((F.width + 15) / 16, (F.height + 7) / 8);
    k_count_paths<<<grid, 128, 0, st>>>(S, F, totals);
    return cudaGetLastError();
}

cudaError_t launch_render_plain(const DevScene &S, const ExactView &X, const FrameParams &F, float4 *accum,
                                uchar4 *display, float4 *frame, cudaStream_t st) {
    dim3 grid((F.width + 15) / 16, (F.height + 7) / 8);
    if (X.on)
        k_render_plain<true><<<grid, 128, size_t(kSharedStack) * 128 * sizeof(uint2), st>>>(S, X, F, accum, display, frame);
    else
        k_render_plain<false><<<grid, 128, 0, st>>>(S, X, F, accum, display, frame);
    return cudaGetLastError();
}

}  // namespace ae
