// exact_trace.cuh - the reference's traversals answered on the optimised
// structures, with the reference's own answer guaranteed ray by ray.
//
// The plain walks (traverse_ref, the deferred shader's traverse_bounded and
// occluded) visit a binary tree in a prescribed order.  What they return does
// not depend on most of that order:
//
//   * A triangle or object ("candidate") is accepted when the slab tests of
//     all boxes above it pass at the time and its own t is at most the nearest
//     accepted so far.  The slab test's arithmetic is monotone in the box, so
//     it passes for a box whenever it passes for a box inside it.
//   * Let w be the candidate of smallest t among a set C that holds every
//     candidate the walk could accept, and let the next smallest t in C lie
//     beyond t_w (1 + 2^-14) ("the band").  Whenever the walk reaches w, the
//     nearest accepted distance is still beyond the band.  So if the slab
//     tests above w pass with the end of the band as their far bound, w is
//     accepted, and nothing can replace it: w is the answer, whatever the
//     visiting order and whatever happens to the other candidates.
//
// C: an accepted triangle's hit point o + d t lies within
// eps = A 2^-17 (|o| + R) of the triangle, A = |e1| |e2| / |e1 x e2| at most over the
// scene's triangles and its planar objects (by their edges): the binary32 errors of the plane distance and of the
// barycentric test (both under 2^-21 (|o| + R) in the plane's normal, that times
// A within the plane), with a factor of eight to spare.  The walk here widens
// every box by eps (4 eps in world space, which covers the instance
// transforms too), prunes with the band's end, and so enumerates C.
//
// An accepted sphere's point lies off the sphere by up to 2^-21 D^2 / r, D the
// larger of r and the distance of origin and centre: the discriminant's
// terms, each of D^2 |d|^2, are rounded 16 times (2^-24 each), and the square
// root of r^2 + x is at most r + x / 2r.  World boxes are widened by four times
// that, taken over the spheres with D <= |o| + |c| + r, which is a quadratic in
// |o| (sphere_a and so on).  Rays for which this exceeds 2^-8 of the scene (tiny
// spheres seen from far) are walked by the reference walk.  One bound from the
// scene's size and the smallest radius would not do: beside a ground sphere of
// 1,000 it widens every box past all 484 spheres of 0.2 on it (486 objects a
// ray instead of 2.2).
//
// The slab tests above w: in the mesh, the triangle's own bounding box lies
// inside every node above it (the build checks that, leaf_enclosed in
// fast_build.cu; the walks are off for a scene with a tree where it does not);
// in the instance tree, `chain` holds the
// intersection of all boxes above the object (flat leaves are widened beyond
// their parents, so the leaf's box alone would not do).
//
// A ray for which any of this does not hold - two candidates within the band
// (a hit on a shared edge, coincident surfaces), a grazed box, a direction
// with a zero component - is walked by the reference walk itself.
//
// Against the reference walks, whose binary float boxes cost two loads and two
// slab tests a node and whose order finds far hits first: 200,003 visibility
// segments 1290 -> 370 us (kernels); 960x540 hybrid frames of 260 objects,
// G-buffer 0.81 -> 0.36 ms, resolve 3.3 -> 2.2 ms; 480x270 compute-only frames
// of 66 objects and 59,398 triangles 2062 -> 584 us.  They are bound as
// closest_fast is: instruction issue and divergence, not bytes.
#pragma once
#include "fast_trace.cuh"
#include "shade.cuh"

namespace ae {

struct ExactView {
    FastView V;
    const float4 *chain;       // per object slot: box minimum, box maximum
    float k;                   // A 2^-17
    float world_r, mesh_r;     // largest coordinates in world space and in any mesh's space
    float sphere_a, sphere_b, sphere_c;  // 2^-19 (max 1/r, 2 max q/r, max q^2/r), 0 without spheres
    float max_origin;          // rays from farther out (1-norm) are left to the reference walk
    uint32_t on;               // 0: the scene needs the reference walk (see exact_view)
};

constexpr float kBand = 1.00006103515625f;  // 1 + 2^-14

AE_DEV float norm1(f3 v) { return fabsf(v.x) + fabsf(v.y) + fabsf(v.z); }
AE_DEV float world_eps(const ExactView &X, f3 o) {
    const float n = norm1(o);
    return fmaf(fmaf(X.sphere_a, n, X.sphere_b), n, X.sphere_c) + 4.0f * X.k * (n + X.world_r);
}
AE_DEV f3 widening(float eps, f3 inv) { return eps * mk(fabsf(inv.x), fabsf(inv.y), fabsf(inv.z)); }
// Components for which 1/d and its products with box distances stay finite
// and away from the 0 * inf of the slab test.
AE_DEV bool plain_direction(f3 d) {
    const float lo = fminf(fminf(fabsf(d.x), fabsf(d.y)), fabsf(d.z));
    return lo > 1e-20f && fabsf(d.x) < 1e20f && fabsf(d.y) < 1e20f && fabsf(d.z) < 1e20f;  // false for NaN
}

// The reference's slab test over a triangle's bounding box.
AE_DEV bool triangle_box_passes(const float4 *r, f3 o, f3 d, float tn, float far) {
    const float4 r0 = __ldg(r), r1 = __ldg(r + 1), r2 = __ldg(r + 2);
    const f3 p0 = mk(r0.x, r0.y, r0.z), p1 = mk(r0.w, r1.x, r1.y), p2 = mk(r1.z, r1.w, r2.x);
    return plain_direction(d) && slab_ref(o, 1.0f / d, vmin(vmin(p0, p1), p2), vmax(vmax(p0, p1), p2), tn, far);
}
AE_DEV bool chain_passes(const ExactView &X, uint32_t object, f3 o, f3 d, float tn, float far) {
    const float4 lo = __ldg(X.chain + 2 * object), hi = __ldg(X.chain + 2 * object + 1);
    return slab_ref(o, 1.0f / d, mk(lo.x, lo.y, lo.z), mk(hi.x, hi.y, hi.z), tn, far);
}

// Nothing in the ray is NaN, infinite or negative where the walks' arithmetic
// counts on it (a user's ray may be anything).
AE_DEV bool plain_ray(const ExactView &X, f3 o, f3 d, float time, float tn, float far) {
    return plain_direction(d) && norm1(o) <= X.max_origin && fabsf(time) < 1e30f && tn >= 0.0f && tn < 1e30f && far < 1e30f &&
           far == far;
}

struct MeshRay {
    f3 o, d;
    uint32_t root, tri_base;
};
AE_DEV MeshRay to_mesh(const FastView &V, uint32_t instance, f3 o, f3 d) {
    // ToLocal (hybrid:534-543), as trace_mesh.
    const float4 *ip = reinterpret_cast<const float4 *>(V.inst + instance);
    const float4 a = __ldg(ip), b = __ldg(ip + 1), c = __ldg(ip + 2);
    MeshRay r;
    r.o = quat_rotate(-b.x, -b.y, -b.z, b.w, o - mk(a.x, a.y, a.z)) * c.z;
    r.d = quat_rotate(-b.x, -b.y, -b.z, b.w, d) * c.z;
    r.root = __float_as_uint(c.x);
    r.tri_base = __float_as_uint(c.y);
    return r;
}

// Which objects a walk tests: all, those the rasterizer draws (meshes and
// raster proxies), or the others.
enum { kAllObjects = 0, kRasterObjects = 1, kTracedObjects = 2 };

// IsRasterProxy, deferred:1011-1017 (renderer/renderer.h:317-323).
AE_DEV bool is_raster_proxy(const ae_object *obj, const ObjHead &hd) {
    return hd.shape == AE_SHAPE_BOX && hd.material != AE_MAT_ISOTROPIC && hd.texture == AE_NO_TEXTURE &&
           ld4(reinterpret_cast<const char *>(obj) + 64).w == 0.0f;
}

enum { kExactMiss = 0, kExactHit = 1, kUndecided = 2 };

// Closest hit before `lim` of a walk that starts with the far bound `far`
// (lim <= far; equal where the caller asks for the closest hit itself).  A hit
// in `best`, kExactMiss when the walk's closest hit does not lie before lim, or
// kUndecided: ask the reference walk.
template <int OBJECTS, int SS>
AE_DEV int closest_exact(const DevScene &S, const ExactView &X, f3 o, f3 d, float time, float tn, float lim, float far,
                         Best &best, uint2 *stk, int tid, int nt) {
    const FastView &V = X.V;
    best.t = lim; best.alpha = 0.0f; best.beta = 0.0f;
    best.object = AE_MISS; best.prim = AE_MISS; best.lrank = 0;
    if (V.troot == kEmptyTlas) return kExactMiss;
    if (!plain_ray(X, o, d, time, tn, lim) || !(far >= lim)) return kUndecided;
    float second = 3.402823466e38f;
    WalkStack<SS> K;
    int sp = 0, base = -1;
    uint32_t cur = V.troot, slot = 0, tri_base = 0;
    f3 lo = o, ld = d;
    f3 inv = mk(slab_inv(d.x), slab_inv(d.y), slab_inv(d.z));
    f3 e = widening(world_eps(X, o), inv);
    for (;;) {
        bool have = true;
        while (!(cur & kLeafBit)) {
            float tm[4];
            uint32_t ch[4];
            child_test<true>((base < 0 ? V.tnodes : V.nodes) + cur, lo, inv, e, tn, best.t * kBand, tm, ch);
            if (sort_hits(tm, ch)) {
                push_far(K, stk, sp, tid, nt, tm, ch);
                cur = ch[0];
                continue;
            }
            have = false;
            break;
        }
        if (have && base >= 0) {
            const uint32_t first = leaf_first(cur), cnt = leaf_count(cur);
            for (uint32_t j = 0; j < cnt; j++) {
                const float4 *r = V.tris + 3 * (size_t(tri_base) + first + j);
                float t, a, b;
                if (!tri_test_ref(lo, ld, tn, best.t * kBand, __ldg(r), __ldg(r + 1), __ldg(r + 2), t, a, b)) continue;
                if (t < best.t) {
                    if (best.object != AE_MISS) second = best.t;
                    best.t = t; best.alpha = a; best.beta = b;
                    best.object = slot; best.prim = first + j;
                } else {
                    second = fminf(second, t);
                }
            }
        } else if (have) {
            const uint32_t s = leaf_first(cur);
            const uint4 m = __ldg(V.meta + s);
            const uint32_t shape = m.x & 0xffu;
            const ae_object *obj = S.objects + s;
            if (shape == AE_SHAPE_MESH) {
                if (OBJECTS != kTracedObjects) {
                    slot = s;
                    const MeshRay mr = to_mesh(V, m.y, o, d);
                    lo = mr.o; ld = mr.d;
                    inv = mk(slab_inv(ld.x), slab_inv(ld.y), slab_inv(ld.z));
                    e = widening(X.k * (norm1(lo) + X.mesh_r), inv);
                    tri_base = mr.tri_base;
                    cur = mr.root;
                    base = sp;
                    continue;
                }
            } else if (OBJECTS == kAllObjects ||
                       (is_raster_proxy(obj, load_head(obj)) == (OBJECTS == kRasterObjects))) {
                DHit h;
                bool hit;
                const float tf = best.t * kBand;
                if (shape == AE_SHAPE_SPHERE) hit = hit_sphere_ref(obj, o, d, time, tn, tf, h);
                else if (shape == AE_SHAPE_QUAD) hit = hit_planar_ref(obj, false, o, d, tn, tf, h);
                else if (shape == AE_SHAPE_TRIANGLE) hit = hit_planar_ref(obj, true, o, d, tn, tf, h);
                else hit = hit_box_ref(obj, o, d, tn, tf, h);
                if (hit && h.t < best.t) {
                    if (best.object != AE_MISS) second = best.t;
                    best.t = h.t; best.alpha = h.alpha; best.beta = h.beta;
                    best.object = s; best.prim = AE_MISS;
                } else if (hit) {
                    second = fminf(second, h.t);
                }
            }
        }
        // Next entry within the band; one below `base` leads back to the
        // instance tree.
        bool found = false;
        const float end = best.t * kBand;
        while (sp > 0 && !found) {
            sp--;
            const uint2 n = stack_at(K, stk, sp, tid, nt);
            cur = n.x;
            found = __uint_as_float(n.y) <= end * kExitGrow;
        }
        if (!found) break;
        if (sp < base) {
            base = -1;
            lo = o;
            inv = mk(slab_inv(d.x), slab_inv(d.y), slab_inv(d.z));
            e = widening(world_eps(X, o), inv);
        }
    }
    if (best.object == AE_MISS) return second <= lim ? kUndecided : kExactMiss;
    const float end = fminf(best.t * kBand, far);
    if (second <= best.t * kBand || !chain_passes(X, best.object, o, d, tn, end)) return kUndecided;
    if (best.prim != AE_MISS) {
        const MeshRay mr = to_mesh(V, __ldg(&V.meta[best.object].y), o, d);
        if (!triangle_box_passes(V.tris + 3 * (size_t(mr.tri_base) + best.prim), mr.o, mr.d, tn, end)) return kUndecided;
    }
    return kExactHit;
}

// Whether any candidate of the any-hit walk (deferred:1115-1171: glass and
// lights do not block; far stays tf) is accepted: kExactHit, kExactMiss, or
// kUndecided when a candidate was found but none whose boxes surely pass.
template <int SS>
AE_DEV int occluded_exact(const DevScene &S, const ExactView &X, f3 o, f3 d, float time, float tn, float tf, uint2 *stk,
                          int tid, int nt) {
    const FastView &V = X.V;
    if (V.troot == kEmptyTlas) return kExactMiss;
    if (!plain_ray(X, o, d, time, tn, tf)) return kUndecided;
    bool unsure = false;
    WalkStack<SS> K;
    int sp = 0, base = -1;
    uint32_t cur = V.troot, slot = 0, tri_base = 0;
    f3 lo = o, ld = d;
    f3 inv = mk(slab_inv(d.x), slab_inv(d.y), slab_inv(d.z));
    f3 e = widening(world_eps(X, o), inv);
    for (;;) {
        bool have = true;
        while (!(cur & kLeafBit)) {
            float tm[4];
            uint32_t ch[4];
            child_test<true>((base < 0 ? V.tnodes : V.nodes) + cur, lo, inv, e, tn, tf, tm, ch);
            if (sort_hits(tm, ch)) {
                push_far(K, stk, sp, tid, nt, tm, ch);
                cur = ch[0];
                continue;
            }
            have = false;
            break;
        }
        if (have && base >= 0) {
            const uint32_t first = leaf_first(cur), cnt = leaf_count(cur);
            for (uint32_t j = 0; j < cnt; j++) {
                const float4 *r = V.tris + 3 * (size_t(tri_base) + first + j);
                float t, a, b;
                if (!tri_test_ref(lo, ld, tn, tf, __ldg(r), __ldg(r + 1), __ldg(r + 2), t, a, b)) continue;
                if (triangle_box_passes(r, lo, ld, tn, tf) && chain_passes(X, slot, o, d, tn, tf)) return kExactHit;
                unsure = true;
            }
        } else if (have) {
            const uint32_t s = leaf_first(cur);
            const uint4 m = __ldg(V.meta + s);
            const uint32_t shape = m.x & 0xffu, mat = m.x >> 8;
            if (mat != AE_MAT_DIELECTRIC && mat != AE_MAT_DIFFUSE_LIGHT) {
                const ae_object *obj = S.objects + s;
                if (shape == AE_SHAPE_MESH) {
                    slot = s;
                    const MeshRay mr = to_mesh(V, m.y, o, d);
                    lo = mr.o; ld = mr.d;
                    inv = mk(slab_inv(ld.x), slab_inv(ld.y), slab_inv(ld.z));
                    e = widening(X.k * (norm1(lo) + X.mesh_r), inv);
                    tri_base = mr.tri_base;
                    cur = mr.root;
                    base = sp;
                    continue;
                }
                DHit h;
                bool hit;
                if (shape == AE_SHAPE_SPHERE) hit = hit_sphere_ref(obj, o, d, time, tn, tf, h);
                else if (shape == AE_SHAPE_QUAD) hit = hit_planar_ref(obj, false, o, d, tn, tf, h);
                else if (shape == AE_SHAPE_TRIANGLE) hit = hit_planar_ref(obj, true, o, d, tn, tf, h);
                else hit = hit_box_ref(obj, o, d, tn, tf, h);
                if (hit) {
                    if (chain_passes(X, s, o, d, tn, tf)) return kExactHit;
                    unsure = true;
                }
            }
        }
        if (sp == 0) break;
        sp--;
        cur = stack_at(K, stk, sp, tid, nt).x;
        if (sp < base) {
            base = -1;
            lo = o;
            inv = mk(slab_inv(d.x), slab_inv(d.y), slab_inv(d.z));
            e = widening(world_eps(X, o), inv);
        }
    }
    return unsure ? kUndecided : kExactMiss;
}

// A finished hit as the plain walks return it.
AE_DEV void exact_hit_record(const DevScene &S, const Best &b, f3 o, f3 d, float time, DHit &h) {
    ae_hit r;
    r.t = b.t; r.alpha = b.alpha; r.beta = b.beta; r.object = b.object; r.prim = b.prim;
    surface_from_hit(S, r, o, d, time, h);
}

}  // namespace ae
