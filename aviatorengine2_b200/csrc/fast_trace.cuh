// fast_trace.cuh - the optimised closest-hit traversal: data layout (4-wide
// quantised BLAS, leaf-ordered triangle records, per-instance records) and the
// device walk, shared by the closest-hit entry points and the wavefront path
// tracer.  See fast.cu for how the structures are built and why the results
// match the reference's walk.
#pragma once
#include <cuda_runtime.h>

#include <map>
#include <string>
#include <tuple>
#include <vector>

#include "context.h"
#include "trace_common.cuh"

namespace ae {

// A 4-wide node of the walks, 64 bytes.  `scale` holds, per axis, the biased
// binary32 exponent of the node's scale 2^e (bytes 0-2).  A child's eight
// bytes are its quantised planes {lo x, lo y, lo z, hi x, hi y, hi z} and the two
// bytes of kPlaneTail: one byte permute of the pair with a selector that the
// ray's direction sign picks gives the bits 0xc0qq0000, the float -V(q) with
// V(q) = 2 + q/64 below q = 128 and 4 + (q - 128)/32 from there on (the byte
// spans the exponent's last bit and seven bits of the mantissa), and plane q
// lies at o + V(q) 2^e.  So a plane costs one permute and one fma, with no
// conversion and no subtraction of a bias.  An unused slot carries
// kPlaneUnused: read as a float, its second word is +inf instead of a negative
// number, which the interval test takes for an entry distance.
struct QNode {
    float ox, oy, oz;        // frame origin, a little over 2 * 2^e below the node box minimum
    uint32_t scale;
    uint2 plane[4];
    uint32_t child[4];       // interior: node index; leaf: leaf_ref(first, count); kNoChild
};
static_assert(sizeof(QNode) == 64, "QNode must be 64 bytes");
constexpr uint32_t kPlaneTail = 0xc0000000u, kPlaneUnused = 0x7f800000u;  // bytes 6-7 of a child's planes

// The node layout that ae_build_wide_bvh hands out (include/ae_b200.h).
struct WideNode {            // 64 B
    float ox, oy, oz;        // node box minimum
    int8_t ex, ey, ez;       // child box scale 2^e per axis
    uint8_t nchild;          // children in use (2..4)
    uint8_t lo[3][4];        // [axis][child]
    uint8_t hi[3][4];
    uint32_t child[4];       // interior: node index; leaf: leaf_ref(first, count)
    uint32_t pad[2];
};
static_assert(sizeof(WideNode) == 64, "WideNode must be 64 bytes");
constexpr uint32_t kLeafBit = 0x80000000u;
constexpr uint32_t kNoChild = kLeafBit;  // a leaf of count 0
// A leaf reference: bit 31 set, primitive count in bits 24-30 (1..127), first
// slot in bits 0-23.  prepare_fast refuses meshes outside those limits.
constexpr uint32_t kMaxLeafFirst = 1u << 24;
constexpr uint32_t kMaxLeafCount = 127u;
__host__ __device__ inline uint32_t leaf_ref(uint32_t first, uint32_t count) { return kLeafBit | (count << 24) | first; }
__host__ __device__ inline uint32_t leaf_first(uint32_t ref) { return ref & 0x00ffffffu; }
__host__ __device__ inline uint32_t leaf_count(uint32_t ref) { return (ref >> 24) & 0x7fu; }

struct FastInst {            // 48 B
    float px, py, pz, scale;
    float qx, qy, qz, qw;
    uint32_t root;           // QNode index of the mesh root, or a leaf ref
    uint32_t tri_base;       // first triangle record of the mesh
    float inv_scale;         // 1 / scale as ToLocal divides, 1 for a rigid instance
    uint32_t sub;            // the mesh's entry in FastScene::sub_refs
};
static_assert(sizeof(FastInst) == 48, "FastInst must be 48 bytes");

// The instance-level tree of the optimised walks: 4-wide QNodes over every
// object of the scene, one object per leaf (leaf_ref(slot, 1)), boxes from
// conservative world bounds of each object (fast.cu: k_object_boxes) and
// refreshed on the device whenever the instances move.  The ranking of equal
// distances does not depend on this tree: an object's rank comes from the
// reference TLAS leaf that holds it (the metadata's z word).
constexpr uint32_t kEmptyTlas = kLeafBit;  // root of a scene without objects (a leaf of count 0)
constexpr int kTlas4Stack = 40;
// Depth of the BLAS nodes whose boxes bound a mesh for the instance tree: up
// to 2^kSubBoxDepth local boxes per mesh, each corner through the instance
// transform.
constexpr int kSubBoxDepth = 8;

struct FastScene {
    DevBuf<QNode> nodes;
    DevBuf<float4> tris;     // 3 float4 per triangle
    DevBuf<FastInst> inst;
    DevBuf<uint4> obj_meta;  // per object slot, see FastView::meta
    DevBuf<uint4> shade16;   // precision form: FP16 normals and UVs, 2 per triangle
    uint32_t shade16_tris = 0;
    // Ray counters of the batch walker (k_closest_walk), one per launch in
    // flight: a ring, so launches on different streams never share one.
    static constexpr uint32_t kWalkCounters = 64;
    DevBuf<uint32_t> walk_next;
    uint32_t walk_pos = 0;
    uint32_t n_nodes = 0, n_tris = 0;
    int max_stack = 0;
    uint64_t geometry_key = ~0ull, scene_key = ~0ull;
    bool has_volumes = false;
    // a mesh is listed (mesh_roots) whose structures are not on the device yet
    // (a build that failed is retried by the next prepare_fast)
    bool geometry_dirty = false;
    // per distinct mesh (vertexBase, indexBase, triangleCount, blasBase)
    std::map<std::tuple<uint32_t, uint32_t, uint32_t, uint32_t>, std::pair<uint32_t, uint32_t>> mesh_roots;
    // Instance-level tree.  Per mesh: its local sub-boxes (host_sub, six
    // floats each) at sub_boxes[first .. first + count) and the largest
    // coordinate magnitude they reach.
    struct MeshSub {
        uint32_t first, count, index;
        float radius;
    };
    std::map<std::tuple<uint32_t, uint32_t, uint32_t, uint32_t>, MeshSub> mesh_sub;
    std::vector<float> host_sub;
    DevBuf<float> sub_boxes;
    DevBuf<uint2> sub_refs;       // per mesh: its first sub-box and their number
    DevBuf<QNode> tnodes;         // the tree's nodes (boxes rewritten on every refresh)
    DevBuf<float> tbox;           // float box per tree node (6 floats)
    DevBuf<float> obj_box;        // conservative world box per object (6 floats)
    DevBuf<float> static_box;     // analytic objects' boxes (6 floats per object slot)
    DevBuf<int32_t> tlevels;      // tree nodes by depth, deepest first
    DevBuf<uint32_t> tflag;       // set by the refresh when a box cannot be quantised
    std::vector<int32_t> tlevel_start;
    DevBuf<int32_t> tlevel_start_dev;
    std::vector<float> inst_radius;  // per instance: its mesh's largest local coordinate
    uint32_t troot = kEmptyTlas, n_tnodes = 0;
    // What the exact walks need beyond (exact_trace.cuh): the shape factor A of
    // the meshes' triangles and of the planar objects, the largest mesh-space coordinate, and per object the
    // intersection of the reference TLAS boxes above it.
    float tri_factor = 1.0f, planar_factor = 1.0f, mesh_range = 0.0f, range = 1.0f;
    bool loose_trees = false;  // a triangle reaches out of a box above it in its tree
    bool odd_boxes = false;    // an object has no box that is sure to hold it (build_instance_tree)
    double sphere[3] = {};     // largest 1/r, q/r and q^2/r over the spheres, q = |centre| + r
    uint2 nan_ref = {0xffffffffu, 0xffffffffu}, nan_wt = {0xffffffffu, 0xffffffffu};
    DevBuf<float4> obj_chain;
    DevBuf<int32_t> tlas_parent;
    int tlas_stack = 0;
    float static_range = 0.0f;    // largest coordinate magnitude of the analytic objects' boxes
    uint64_t tlas_key = ~0ull, sub_key = ~0ull;
};

// Traversal stack per thread, one for both trees (a mesh's entries lie above
// the instance tree's): the first kSharedStack entries in shared memory, the
// rest (rarely reached: only along the deepest paths of the largest meshes) in
// a per-thread local array.  prepare_fast checks that no mesh tree needs more
// than kFastStack entries and no instance tree more than kTlas4Stack.
constexpr int kSharedStack = 12;
constexpr int kFastStack = 64;
constexpr int kWalkStack = kFastStack + kTlas4Stack;

// ---------------------------------------------------------------------------
// Device
// ---------------------------------------------------------------------------
struct FastView {
    const QNode *nodes;
    const float4 *tris;
    const FastInst *inst;
    const uint4 *meta;      // x: shape | material << 8, y: instance, z: first slot of its reference TLAS leaf,
                            // w: that leaf's node
    const QNode *tnodes;    // instance-level tree
    uint32_t troot;         // its root: a node index, leaf_ref(slot, 1), or kEmptyTlas
    // What the reference walk answers a ray whose direction is NaN on every axis
    // (a path that met a degenerate normal), by triangle test: (object slot,
    // triangle slot), AE_MISS for none.  See nan_answers in fast.cu.
    uint2 nan_ref, nan_wt;
};

// The view of a prepared scene; `inst` and `tnodes` may name another copy of
// the per-frame arrays (serving frame sets).
inline FastView fast_view(const FastScene &F, const FastInst *inst = nullptr, const QNode *tnodes = nullptr) {
    return FastView{F.nodes.ptr, F.tris.ptr, inst ? inst : F.inst.ptr, F.obj_meta.ptr, tnodes ? tnodes : F.tnodes.ptr,
                    F.troot, F.nan_ref, F.nan_wt};
}

// Best candidate so far.  Equal distances rank by (object rank, leaf rank,
// slot), larger meaning visited later by the reference's walk (see the file
// comment): an object's rank is ~first slot of the reference TLAS leaf holding
// it (the metadata's z word), then its slot; the leaf rank is ~first slot of
// the BLAS leaf.  Object ranks are read when two distances are equal, which is
// rare, and not carried along.
struct Best {
    float t, alpha, beta;
    uint32_t object, prim;
    uint32_t lrank;
};
AE_DEV bool later_object(const FastView &V, uint32_t object, uint32_t than) {
    if (than == AE_MISS) return true;
    const uint32_t a = __ldg(&V.meta[object].z), b = __ldg(&V.meta[than].z);
    return a != b ? a < b : object > than;
}
// Given a hit at t <= best.t (the tests reject t > far), keep it if nearer or
// equally near and later in the reference's visit order.
AE_DEV bool takes(const FastView &V, const Best &b, float t, uint32_t object, uint32_t lrank, uint32_t slot) {
    if (t < b.t) return true;
    if (object != b.object) return later_object(V, object, b.object);
    if (lrank != b.lrank) return lrank > b.lrank;
    return slot > b.prim;
}

// A ray without a direction: its answer is the scene's, and known.
AE_DEV bool no_direction(f3 d) { return d.x != d.x && d.y != d.y && d.z != d.z; }
template <bool WT>
AE_DEV void nan_best(const FastView &V, Best &b) {
    const uint2 h = WT ? V.nan_wt : V.nan_ref;
    if (h.x == AE_MISS) return;
    const float nan = __int_as_float(0x7fffffff);
    const bool sphere = (__ldg(&V.meta[h.x].x) & 0xffu) == AE_SHAPE_SPHERE;
    b.t = nan;
    b.alpha = b.beta = sphere ? 0.0f : nan;
    b.object = h.x;
    b.prim = h.y;
}

// HitMeshTriangle (hybrid:564-598), correctly rounded; p1/p2 give e1/e2 by the
// same subtraction the reference performs.
AE_DEV bool tri_test_ref(f3 o, f3 d, float tn, float tf, const float4 &r0, const float4 &r1, const float4 &r2,
                         float &t, float &a, float &b) {
    const f3 p0 = mk(r0.x, r0.y, r0.z), p1 = mk(r0.w, r1.x, r1.y), p2 = mk(r1.z, r1.w, r2.x);
    const f3 e1 = p1 - p0, e2 = p2 - p0;
    const f3 n = cross(e1, e2);
    const float nn = dot(n, n);
    if (nn < 1e-12f) return false;
    const float den = dot(n, d);
    if (AE_FABS(den) < 1e-12f) return false;
    t = AE_DIV(AE_SUB(dot(n, p0), dot(n, o)), den);
    if (t < tn || t > tf) return false;
    const f3 pl = o + d * t - p0;
    const f3 ca = cross(pl, e2), cb = cross(e1, pl);
    // Most candidates lie outside by far more than rounding: those are turned
    // away without the reference's three divisions.  a = (n / nn) . ca and
    // its terms' roundings stay within 2^-21 of sum |n_i ca_i| / nn (and of
    // the smallest binary32 values, which the last term covers), so a sum
    // below -2^-20 of that has a < 0; the same for b, and for a + b > 1.
    const float ma = fmaf(fabsf(n.x), fabsf(ca.x), fmaf(fabsf(n.y), fabsf(ca.y), fabsf(n.z * ca.z)));
    const float mb = fmaf(fabsf(n.x), fabsf(cb.x), fmaf(fabsf(n.y), fabsf(cb.y), fabsf(n.z * cb.z)));
    const float sa = fmaf(n.x, ca.x, fmaf(n.y, ca.y, n.z * ca.z)), sb = fmaf(n.x, cb.x, fmaf(n.y, cb.y, n.z * cb.z));
    constexpr float kRel = 9.5367431640625e-07f;  // 2^-20
    const float tiny = nn * 1e-30f;
    if (fmaf(ma, kRel, sa) + tiny < 0.0f || fmaf(mb, kRel, sb) + tiny < 0.0f) return false;
    if (fmaf(ma + mb, -kRel, sa + sb) > fmaf(nn, kRel, nn) + tiny) return false;
    const f3 w = n / nn;
    a = dot(w, ca);
    b = dot(w, cb);
    return !(a < 0.0f || b < 0.0f || AE_ADD(a, b) > 1.0f);
}

// The watertight test (trace_common.cuh) over a 48-byte triangle record.
AE_DEV bool tri_test_wt(f3 o, const WtRay &W, float tn, float tf, const float4 &r0, const float4 &r1,
                        const float4 &r2, float &t, float &a, float &b) {
    return tri_wt(o, W, tn, tf, mk(r0.x, r0.y, r0.z), mk(r0.w, r1.x, r1.y), mk(r1.z, r1.w, r2.x), t, a, b);
}

// Relative widening of slab intervals in the optimised walks: an interval's
// exit and the best distance are scaled up by 1 + 2^-19 before they are
// compared with an entry.  Together with the planes' room (kPlaneRoom,
// quantise.cuh) that covers the rounding of the plane distances: neither a
// nearer hit nor one on a box's face is pruned.
constexpr float kExitGrow = 1.0000019073486328125f;  // 1 + 2^-19

AE_DEV float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
AE_DEV float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Entry distances of a node's four child boxes; +inf for a child that the ray
// misses or that starts beyond the best hit.  Distances are in units of the
// ray parameter: plane q of an axis lies at V(q) 2^e / d + (o - p) / d.
//
// The walks are bound by issue slots with 12-15 of 32 lanes active, so the
// count of instructions here is what a step costs: the permute builds a
// plane's float directly, the near and far bytes are chosen by the permute's
// selector instead of by selects, three-operand min and max fold an interval,
// and an unused slot rejects itself.  NaN distances (a NaN in the ray) drop out
// of min and max, so an axis without a direction bounds nothing.
//
// WIDE: every box is widened by a length whose extent in t is `e` per axis.
template <bool WIDE>
AE_DEV void child_test(const QNode *nodep, f3 o, f3 inv, f3 e, float tn, float tf, float tmin[4], uint32_t child[4]) {
    const uint4 *p = reinterpret_cast<const uint4 *>(nodep);
    const uint4 w0 = __ldg(p), pa = __ldg(p + 1), pb = __ldg(p + 2), cr = __ldg(p + 3);
    const float ix = __uint_as_float(__byte_perm(w0.w, 0u, 0x0444u) >> 1) * -inv.x;
    const float iy = __uint_as_float(__byte_perm(w0.w, 0u, 0x1444u) >> 1) * -inv.y;
    const float iz = __uint_as_float(__byte_perm(w0.w, 0u, 0x2444u) >> 1) * -inv.z;
    const float bx = (__uint_as_float(w0.x) - o.x) * inv.x;
    const float by = (__uint_as_float(w0.y) - o.y) * inv.y;
    const float bz = (__uint_as_float(w0.z) - o.z) * inv.z;
    const float nbx = WIDE ? bx - e.x : bx, nby = WIDE ? by - e.y : by, nbz = WIDE ? bz - e.z : bz;
    const float fbx = WIDE ? bx + e.x : bx, fby = WIDE ? by + e.y : by, fbz = WIDE ? bz + e.z : bz;
    // Selectors {6, 6, q, 7}: q = 0, 1, 2 for the low planes and 3, 4, 5 for
    // the high ones; a negative direction enters through the high plane.
    const uint32_t nx = 0x7066u ^ (uint32_t(__float_as_int(inv.x) >> 31) & 0x300u), fx = nx ^ 0x300u;
    const uint32_t ny = 0x7166u ^ (uint32_t(__float_as_int(inv.y) >> 31) & 0x500u), fy = ny ^ 0x500u;
    const uint32_t nz = 0x7266u ^ (uint32_t(__float_as_int(inv.z) >> 31) & 0x700u), fz = nz ^ 0x700u;
    const float tfg = tf * kExitGrow;
    const uint32_t lo_w[4] = {pa.x, pa.z, pb.x, pb.z}, hi_w[4] = {pa.y, pa.w, pb.y, pb.w};
    child[0] = cr.x; child[1] = cr.y; child[2] = cr.z; child[3] = cr.w;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float t0x = fmaf(__uint_as_float(__byte_perm(lo_w[k], hi_w[k], nx)), ix, nbx);
        const float t0y = fmaf(__uint_as_float(__byte_perm(lo_w[k], hi_w[k], ny)), iy, nby);
        const float t0z = fmaf(__uint_as_float(__byte_perm(lo_w[k], hi_w[k], nz)), iz, nbz);
        const float t1x = fmaf(__uint_as_float(__byte_perm(lo_w[k], hi_w[k], fx)), ix, fbx);
        const float t1y = fmaf(__uint_as_float(__byte_perm(lo_w[k], hi_w[k], fy)), iy, fby);
        const float t1z = fmaf(__uint_as_float(__byte_perm(lo_w[k], hi_w[k], fz)), iz, fbz);
        // -2e37 and below for a slot in use, +inf for an unused one.
        const float slot = __uint_as_float(hi_w[k]) * 1e37f;
        const float lo = max3(max3(t0x, t0y, t0z), tn, slot);
        const float hi = fminf(min3(t1x, t1y, t1z) * kExitGrow, tfg);
        tmin[k] = lo <= hi ? lo : __int_as_float(0x7f800000);
    }
}

AE_DEV void child_hits(const QNode *nodep, f3 o, f3 inv, float tn, float tf, float tmin[4], uint32_t child[4]) {
    child_test<false>(nodep, o, inv, mk(0.0f, 0.0f, 0.0f), tn, tf, tmin, child);
}

// Safe reciprocal for slab tests: a zero component becomes a huge finite
// value of the same sign, so products stay finite (no 0 * inf); a power of two,
// so that a ray in the plane of a box's face is exactly on it.  The hardware
// reciprocal (within 1 ulp) scales an axis's plane distances by at most 2^-23,
// inside the intervals' widening; a correctly rounded quotient cost about ten
// instructions an axis.
AE_DEV float slab_inv(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return fabsf(x) > 1e-20f ? r : copysignf(73786976294838206464.0f, x);  // 2^66
}

// Sorts child_hits' four (distance, child) pairs nearest first (misses carry
// +inf and sort last); false when none was hit.
AE_DEV bool sort_hits(float tm[4], uint32_t ch[4]) {
#define AE_SWAP(i, j)                                            \
    if (tm[j] < tm[i]) {                                         \
        const float tt = tm[i]; tm[i] = tm[j]; tm[j] = tt;       \
        const uint32_t cc = ch[i]; ch[i] = ch[j]; ch[j] = cc;    \
    }
    AE_SWAP(0, 1) AE_SWAP(2, 3) AE_SWAP(0, 2) AE_SWAP(1, 3) AE_SWAP(1, 2)
#undef AE_SWAP
    return tm[0] != __int_as_float(0x7f800000);
}

// One thread's traversal stack: its column of the block's shared-memory part
// and the entries beyond it.
template <int SS>
struct WalkStack {
    uint2 spill[kWalkStack - SS];
};
// The bound check of the spilled part keeps every access inside the array for
// any input (prepare_fast has checked the trees' needs).
template <int SS>
AE_DEV void stack_push(WalkStack<SS> &K, uint2 *stk, int &sp, int tid, int nt, uint32_t ref, float t) {
    const uint2 e = make_uint2(ref, __float_as_uint(t));
    if (sp < SS) stk[sp * nt + tid] = e;
    else if (sp < kWalkStack) K.spill[sp - SS] = e;
    else return;
    sp++;
}
template <int SS>
AE_DEV uint2 stack_at(const WalkStack<SS> &K, const uint2 *stk, int i, int tid, int nt) {
    return i < SS ? stk[i * nt + tid] : K.spill[i - SS];
}
// A node's hit children but the nearest, farthest first.  Written out, so
// that the sorted distances and references stay in registers (a loop over
// them put both arrays in local memory: eight stores a node, the largest
// single cost of the walks).
template <int SS>
AE_DEV void push_far(WalkStack<SS> &K, uint2 *stk, int &sp, int tid, int nt, const float tm[4], const uint32_t ch[4]) {
    const float none = __int_as_float(0x7f800000);
    if (tm[3] != none) stack_push(K, stk, sp, tid, nt, ch[3], tm[3]);
    if (tm[2] != none) stack_push(K, stk, sp, tid, nt, ch[2], tm[2]);
    if (tm[1] != none) stack_push(K, stk, sp, tid, nt, ch[1], tm[1]);
}

// T (optional): touch counters - wide nodes in `blas`, 48-byte triangle
// records in `tris`.  The stack's first `base` entries belong to the caller.
template <bool WT, int SS = kSharedStack>
AE_DEV void trace_mesh(const FastView &V, const FastInst &I, uint32_t slot, f3 o, f3 d, float tn,
                       Best &best, WalkStack<SS> &K, uint2 *stk, const int base, int tid, int nthreads,
                       Touch *T = nullptr) {
    // ToLocal (hybrid:534-543) exactly as the reference, so the local ray and
    // every triangle's t are bit-identical to the plain kernel's.
    f3 lo = quat_rotate(-I.qx, -I.qy, -I.qz, I.qw, o - mk(I.px, I.py, I.pz));
    f3 ld = quat_rotate(-I.qx, -I.qy, -I.qz, I.qw, d);
    // Multiplying by exactly 1 changes nothing, so rigid instances need no branch.
    lo = lo * I.inv_scale;
    ld = ld * I.inv_scale;
    const f3 inv = mk(slab_inv(ld.x), slab_inv(ld.y), slab_inv(ld.z));
    WtRay W;
    if (WT) W = wt_setup(ld);
    const float4 *tris = V.tris + size_t(I.tri_base) * 3;
    int sp = base;
    uint32_t cur = I.root;
    // Next stack entry still no farther than the best hit; false when none.
    auto pop = [&]() {
        while (sp > base) {
            sp--;
            const uint2 e = stack_at(K, stk, sp, tid, nthreads);
            if (__uint_as_float(e.y) <= best.t * kExitGrow) {
                cur = e.x;
                return true;
            }
        }
        return false;
    };
    for (;;) {
        // Interior nodes until this lane holds a leaf; the warp's lanes then
        // test their leaves' triangles together.
        while (!(cur & kLeafBit)) {
            float tm[4];
            uint32_t ch[4];
            if (T) T->blas++;
            child_hits(V.nodes + cur, lo, inv, tn, best.t, tm, ch);
            if (sort_hits(tm, ch)) {
                push_far(K, stk, sp, tid, nthreads, tm, ch);
                cur = ch[0];
            } else if (!pop()) {
                return;
            }
        }
        const uint32_t first = leaf_first(cur), cnt = leaf_count(cur);
        if (T) T->tris += cnt;
        for (uint32_t k = 0; k < cnt; k++) {
            const uint32_t s = first + k;
            const float4 *r = tris + size_t(s) * 3;
            const float4 r0 = __ldg(r), r1 = __ldg(r + 1), r2 = __ldg(r + 2);
            float t, a, b;
            const bool h = WT ? tri_test_wt(lo, W, tn, best.t, r0, r1, r2, t, a, b)
                              : tri_test_ref(lo, ld, tn, best.t, r0, r1, r2, t, a, b);
            if (h && takes(V, best, t, slot, ~first, s)) {
                best.t = t; best.alpha = a; best.beta = b;
                best.object = slot; best.prim = s;
                best.lrank = ~first;
            }
        }
        if (!pop()) return;
    }
}

// Closest hit of one ray over the whole scene: the instance-level tree
// (nearest child first), analytic objects by the reference intersectors,
// meshes by the 4-wide quantised BLAS.  `stk` is this thread's column of the
// block's shared-memory stack.  T (optional) counts the touches: instance-tree
// nodes, object metadata records, instance records, wide BLAS nodes, triangle
// records.  tmax: as Walker::start.
template <bool WT, int SS = kSharedStack>
AE_DEV Best closest_fast(const DevScene &S, const FastView &V, f3 o, f3 d, float tn, float time, uint2 *stk, int tid,
                         int nt, Touch *T = nullptr, float tmax = kFarStart) {
    Best best;
    best.t = tmax; best.alpha = 0.0f; best.beta = 0.0f;
    best.object = AE_MISS; best.prim = AE_MISS; best.lrank = 0;
    if (V.troot == kEmptyTlas) return best;
    if (no_direction(d)) {
        nan_best<WT>(V, best);
        return best;
    }
    const f3 inv = mk(slab_inv(d.x), slab_inv(d.y), slab_inv(d.z));
    WalkStack<SS> K;
    int sp = 0;
    uint32_t cur = V.troot;
    // Next stack entry no farther than the best hit; false when none is left.
    auto pop = [&]() {
        while (sp > 0) {
            sp--;
            const uint2 e = stack_at(K, stk, sp, tid, nt);
            if (__uint_as_float(e.y) <= best.t * kExitGrow) {
                cur = e.x;
                return true;
            }
        }
        return false;
    };
    for (;;) {
        // Inner nodes until this lane holds an object: the lanes of a warp
        // leave this loop together and then enter their objects together
        // (a lane at a node does not wait through another lane's whole mesh).
        bool live = true;
        while (!(cur & kLeafBit)) {
            float tm[4];
            uint32_t ch[4];
            if (T) T->tlas++;
            child_hits(V.tnodes + cur, o, inv, tn, best.t, tm, ch);
            if (sort_hits(tm, ch)) {
                push_far(K, stk, sp, tid, nt, tm, ch);
                cur = ch[0];
            } else if (!pop()) {
                live = false;
                break;
            }
        }
        if (!live) break;
        const uint32_t slot = leaf_first(cur);
        const uint4 m = __ldg(V.meta + slot);
        const uint32_t shape = m.x & 0xff;
        if (T) T->objects++;
        if (shape == AE_SHAPE_MESH) {
            if (T) T->instances++;
            const float4 *ip = reinterpret_cast<const float4 *>(V.inst + m.y);
            const float4 a = __ldg(ip), b = __ldg(ip + 1), c = __ldg(ip + 2);
            FastInst I;
            I.px = a.x; I.py = a.y; I.pz = a.z; I.scale = a.w;
            I.qx = b.x; I.qy = b.y; I.qz = b.z; I.qw = b.w;
            I.root = __float_as_uint(c.x); I.tri_base = __float_as_uint(c.y);
            I.inv_scale = c.z;
            trace_mesh<WT, SS>(V, I, slot, o, d, tn, best, K, stk, sp, tid, nt, T);
        } else {
            DHit h;
            const ae_object *obj = S.objects + slot;
            bool hit;
            if (shape == AE_SHAPE_SPHERE) hit = hit_sphere_ref(obj, o, d, time, tn, best.t, h);
            else if (shape == AE_SHAPE_QUAD) hit = hit_planar_ref(obj, false, o, d, tn, best.t, h);
            else if (shape == AE_SHAPE_TRIANGLE) hit = hit_planar_ref(obj, true, o, d, tn, best.t, h);
            else hit = hit_box_ref(obj, o, d, tn, best.t, h);
            if (hit && takes(V, best, h.t, slot, 0u, 0u)) {
                best.t = h.t; best.alpha = h.alpha; best.beta = h.beta;
                best.object = slot; best.prim = AE_MISS; best.lrank = 0;
            }
        }
        if (!pop()) break;
    }
    return best;
}

}  // namespace ae
