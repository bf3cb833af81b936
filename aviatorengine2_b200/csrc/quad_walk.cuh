// quad_walk.cuh - the nearest hit by four lanes a ray, for launches with few
// rays.
//
// A launch of a few thousand rays lasts as long as its slowest ray's chain of
// steps: node address, load, four child boxes, sort, push, next node.  One
// lane does the four boxes and the sort one after another (about a hundred
// dependent instructions) while the launch leaves most lanes idle.  Here each
// lane of an aligned quad takes one child of every node and one triangle of
// every leaf; the ray, the stack and the best hit so far are the quad's, the same in
// its four lanes.  The hit does not depend on the visiting order (takes()), so
// it is closest_fast's bit for bit.
//
// Random rays through 200 instances, whole call, one lane -> four: 500 rays 65
// -> 55 us, 2,000 92 -> 73 us, 8,000 114 -> 86 us; four 256x256 frames of depth
// 8, by their late bounces: 5.15 -> 4.76 ms.
#pragma once
#include "fast_trace.cuh"

namespace ae {

// Stack entries a quad has in a block's shared memory (kSharedStack entries a
// thread, one less so that neighbouring quads start two banks apart).  A ray
// that needs more is walked by closest_fast.
constexpr int kQuadStack = 4 * kSharedStack - 1;

// Child `ql` of a node, as child_test tests it.
AE_DEV float child_distance(const QNode *nodep, int ql, f3 o, f3 inv, float tn, float tf, uint32_t &child) {
    const uint4 w0 = __ldg(reinterpret_cast<const uint4 *>(nodep));
    const uint2 pl = __ldg(nodep->plane + ql);
    child = __ldg(nodep->child + ql);
    const float ix = __uint_as_float(__byte_perm(w0.w, 0u, 0x0444u) >> 1) * -inv.x;
    const float iy = __uint_as_float(__byte_perm(w0.w, 0u, 0x1444u) >> 1) * -inv.y;
    const float iz = __uint_as_float(__byte_perm(w0.w, 0u, 0x2444u) >> 1) * -inv.z;
    const float bx = (__uint_as_float(w0.x) - o.x) * inv.x;
    const float by = (__uint_as_float(w0.y) - o.y) * inv.y;
    const float bz = (__uint_as_float(w0.z) - o.z) * inv.z;
    const uint32_t nx = 0x7066u ^ (uint32_t(__float_as_int(inv.x) >> 31) & 0x300u), fx = nx ^ 0x300u;
    const uint32_t ny = 0x7166u ^ (uint32_t(__float_as_int(inv.y) >> 31) & 0x500u), fy = ny ^ 0x500u;
    const uint32_t nz = 0x7266u ^ (uint32_t(__float_as_int(inv.z) >> 31) & 0x700u), fz = nz ^ 0x700u;
    const float t0x = fmaf(__uint_as_float(__byte_perm(pl.x, pl.y, nx)), ix, bx);
    const float t0y = fmaf(__uint_as_float(__byte_perm(pl.x, pl.y, ny)), iy, by);
    const float t0z = fmaf(__uint_as_float(__byte_perm(pl.x, pl.y, nz)), iz, bz);
    const float t1x = fmaf(__uint_as_float(__byte_perm(pl.x, pl.y, fx)), ix, bx);
    const float t1y = fmaf(__uint_as_float(__byte_perm(pl.x, pl.y, fy)), iy, by);
    const float t1z = fmaf(__uint_as_float(__byte_perm(pl.x, pl.y, fz)), iz, bz);
    const float slot = __uint_as_float(pl.y) * 1e37f;
    const float lo = max3(max3(t0x, t0y, t0z), tn, slot);
    const float hi = fminf(min3(t1x, t1y, t1z) * kExitGrow, tf * kExitGrow);
    return lo <= hi ? lo : __int_as_float(0x7f800000);
}

// The quad's walk; false when its stack ran out (best is then not the
// answer).  stk: the quad's kQuadStack entries.  The four lanes call it
// together with the same arguments.
template <bool WT>
AE_DEV bool walk_quad(const DevScene &S, const FastView &V, f3 o, f3 d, float tn, float time, float tmax, uint2 *stk,
                      Best &best) {
    const int ql = int(threadIdx.x & 3u);
    const uint32_t quad = 0xfu << (threadIdx.x & 28u);
    const float none = __int_as_float(0x7f800000);
    best.t = tmax; best.alpha = 0.0f; best.beta = 0.0f;
    best.object = AE_MISS; best.prim = AE_MISS; best.lrank = 0;
    if (V.troot == kEmptyTlas) return true;
    const f3 tinv = mk(slab_inv(d.x), slab_inv(d.y), slab_inv(d.z));
    // The tree that is walked: its nodes and the ray in its space.
    const QNode *nodes = V.tnodes;
    f3 lo = o, ld = d, inv = tinv;
    WtRay W;
    uint32_t cur = V.troot, tri_base = 0, slot = 0;
    int sp = 0, base = -1;  // base: the instance tree's entries while a mesh is walked, else -1
    for (;;) {
        bool have = true;
        while (!(cur & kLeafBit)) {
            uint32_t child;
            const float t = child_distance(nodes + cur, ql, lo, inv, tn, best.t, child);
            const float a = __shfl_xor_sync(quad, t, 1), b = __shfl_xor_sync(quad, t, 2), c = __shfl_xor_sync(quad, t, 3);
            // How many children come before this one: nearer, or as near and of a lower number.
            const int rank = int(a < t || (a == t && (ql & 1))) + int(b < t || (b == t && (ql & 2))) +
                             int(c < t || (c == t && (ql & 2)));
            const int hits = int(t != none) + int(a != none) + int(b != none) + int(c != none);
            if (hits == 0) {
                have = false;
                break;
            }
            if (sp + hits - 1 > kQuadStack) {
                __syncwarp(quad);  // the lanes' pushes before the caller's walk takes the entries over
                return false;
            }
            if (t != none && rank > 0) stk[sp + hits - 1 - rank] = make_uint2(child, __float_as_uint(t));
            sp += hits - 1;
            const uint32_t first = __ballot_sync(quad, rank == 0) & quad;
            cur = __shfl_sync(quad, child, __ffs(int(first)) - 1);
        }
        if (have && base >= 0) {
            const uint32_t first = leaf_first(cur), cnt = leaf_count(cur);
            bool found = false;
            for (uint32_t k = uint32_t(ql); k < cnt; k += 4) {
                const uint32_t s = first + k;
                const float4 *r = V.tris + (size_t(tri_base) + s) * 3;
                const float4 r0 = __ldg(r), r1 = __ldg(r + 1), r2 = __ldg(r + 2);
                float t, a, b;
                const bool h = WT ? tri_test_wt(lo, W, tn, best.t, r0, r1, r2, t, a, b)
                                  : tri_test_ref(lo, ld, tn, best.t, r0, r1, r2, t, a, b);
                if (h && takes(V, best, t, slot, ~first, s)) {
                    best.t = t; best.alpha = a; best.beta = b;
                    best.object = slot; best.prim = s;
                    best.lrank = ~first;
                    found = true;
                }
            }
            if (__any_sync(quad, found)) {
                // The quad's best of its lanes' four.
                for (int m = 1; m < 4; m <<= 1) {
                    Best x;
                    x.t = __shfl_xor_sync(quad, best.t, m);
                    x.alpha = __shfl_xor_sync(quad, best.alpha, m);
                    x.beta = __shfl_xor_sync(quad, best.beta, m);
                    x.object = __shfl_xor_sync(quad, best.object, m);
                    x.prim = __shfl_xor_sync(quad, best.prim, m);
                    x.lrank = __shfl_xor_sync(quad, best.lrank, m);
                    if (x.object != AE_MISS && x.t <= best.t && takes(V, best, x.t, x.object, x.lrank, x.prim)) best = x;
                }
            }
        } else if (have) {
            const uint32_t s = leaf_first(cur);
            const uint4 m = __ldg(V.meta + s);
            const uint32_t shape = m.x & 0xffu;
            if (shape == AE_SHAPE_MESH) {
                // ToLocal (hybrid:534-543), as trace_mesh.
                const float4 *ip = reinterpret_cast<const float4 *>(V.inst + m.y);
                const float4 a = __ldg(ip), b = __ldg(ip + 1), c = __ldg(ip + 2);
                slot = s;
                lo = quat_rotate(-b.x, -b.y, -b.z, b.w, o - mk(a.x, a.y, a.z)) * c.z;
                ld = quat_rotate(-b.x, -b.y, -b.z, b.w, d) * c.z;
                inv = mk(slab_inv(ld.x), slab_inv(ld.y), slab_inv(ld.z));
                if (WT) W = wt_setup(ld);
                tri_base = __float_as_uint(c.y);
                cur = __float_as_uint(c.x);
                nodes = V.nodes;
                base = sp;
                continue;
            }
            DHit h;
            const ae_object *obj = S.objects + s;
            bool hit;
            if (shape == AE_SHAPE_SPHERE) hit = hit_sphere_ref(obj, o, d, time, tn, best.t, h);
            else if (shape == AE_SHAPE_QUAD) hit = hit_planar_ref(obj, false, o, d, tn, best.t, h);
            else if (shape == AE_SHAPE_TRIANGLE) hit = hit_planar_ref(obj, true, o, d, tn, best.t, h);
            else hit = hit_box_ref(obj, o, d, tn, best.t, h);
            if (hit && takes(V, best, h.t, s, 0u, 0u)) {
                best.t = h.t; best.alpha = h.alpha; best.beta = h.beta;
                best.object = s; best.prim = AE_MISS; best.lrank = 0;
            }
        }
        // Next entry no farther than the best hit; one below `base` leads back
        // to the instance tree.  The lanes' pushes before, their reads after.
        __syncwarp(quad);
        const float far = best.t * kExitGrow;
        bool found = false;
        while (sp > 0 && !found) {
            const uint2 e = stk[--sp];
            cur = e.x;
            found = __uint_as_float(e.y) <= far;
        }
        __syncwarp(quad);
        if (!found) return true;
        if (sp < base) {
            base = -1;
            nodes = V.tnodes;
            lo = o;
            inv = tinv;
        }
    }
}

// closest_fast's answer for the ray that the four lanes of a quad hold.  stk
// is the block's shared-memory stack (kSharedStack entries a thread).
template <bool WT>
AE_DEV Best closest_quad(const DevScene &S, const FastView &V, f3 o, f3 d, float tn, float time, uint2 *stk,
                         float tmax = kFarStart) {
    uint2 *mine = stk + (threadIdx.x >> 2) * kQuadStack;
    // Rays whose arithmetic may overflow to NaN distances, for which the
    // visiting order matters, keep closest_fast's.
    const float size = fabsf(o.x) + fabsf(o.y) + fabsf(o.z) + fabsf(d.x) + fabsf(d.y) + fabsf(d.z) + fabsf(tn) + fabsf(time);
    Best best;
    if (size < 1e15f && tmax == tmax && walk_quad<WT>(S, V, o, d, tn, time, tmax, mine, best)) return best;
    return closest_fast<WT, kQuadStack / 4>(S, V, o, d, tn, time, mine, int(threadIdx.x & 3u), 4, nullptr, tmax);
}

}  // namespace ae
