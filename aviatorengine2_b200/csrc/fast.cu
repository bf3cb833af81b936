// fast.cu - the optimised closest-hit path.
//
// Data layout (built once per geometry upload, in HBM):
//   * per distinct mesh, a 4-wide BVH collapsed from the reference's binary
//     BLAS (scene/bvh.h).  Collapsing only merges interior nodes, so every
//     leaf - and therefore every triangle slot - is the reference's.  A node
//     is 64 bytes: a frame (origin, one power-of-two scale per axis) and four
//     child boxes quantised to 8 bits, rounded outward so a decoded box always
//     contains the exact one (no hit can be lost); built on the device
//     (fast_build.cu, quantise.cuh);
//   * triangles in leaf-slot order as 48-byte records {p0, p1, p2}: one
//     contiguous read per leaf instead of an index fetch plus three vertex
//     fetches;
//   * per instance a 48-byte record with the transform and the mesh's node
//     and triangle bases.
//
// Traversal is nearest-child-first with the far children on one stack for
// both trees (its first entries in shared memory) that also stores each entry's entry distance, so a popped subtree
// farther than the current hit is skipped without touching its node.
//
// Equal distances: the reference's depth-first walk (hybrid:862-917,
// 617-652) accepts a hit at t == far, so of several hits at the same t the one
// visited LAST wins.  Its walk pops the right child first, and the builder
// gives right subtrees the higher leaf slots, so the visit order is: leaves by
// DESCENDING first slot, primitives within a leaf by ascending slot, objects
// before their triangles.  The kernels rank every candidate by that order and
// keep the highest rank among equal t, which reproduces the reference's answer
// whatever order they visit in.
//
// The triangle test is the reference's HitMeshTriangle (hybrid:564-598) in
// correctly rounded binary32, so t and the barycentrics are bit-identical to
// the plain kernel's; the watertight variant (Woop, Benthin and Wald, "Watertight
// Ray/Triangle Intersection", JCGT 2013) is selected with `quant`.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cmath>
#include <cstring>
#include <map>
#include <string>
#include <tuple>
#include <vector>

#include "context.h"
#include "exact_trace.cuh"
#include "quad_walk.cuh"
#include "fast.h"
#include "fast_trace.cuh"
#include "fast_walk.cuh"
#include "kernels.h"
#include "quantise.cuh"
#include "trace_common.cuh"

namespace ae {

// ---------------------------------------------------------------------------
// Host: 4-wide collapse and quantisation
// ---------------------------------------------------------------------------
namespace {

struct Box {
    float lo[3], hi[3];
};
static_assert(sizeof(Box) == 24, "the device's boxes");
Box node_box(const ae_bvh_node &n) { return Box{{n.min_x, n.min_y, n.min_z}, {n.max_x, n.max_y, n.max_z}}; }
// Not inside out, and no coordinate beyond `reach`, infinite or NaN.
bool box_within(const Box &b, float reach) {
    for (int a = 0; a < 3; a++)
        if (!(b.lo[a] <= b.hi[a] && b.lo[a] > -reach && b.hi[a] < reach)) return false;
    return true;
}
float half_area(const Box &b) {
    const float dx = b.hi[0] - b.lo[0], dy = b.hi[1] - b.lo[1], dz = b.hi[2] - b.lo[2];
    return dx * dy + dy * dz + dz * dx;
}

// Smallest exponent e with (extent / 2^e) <= 255, i.e. 8 bits cover the box.
int axis_exponent(float extent) {
    if (!(extent > 0.0f)) return -126;
    int e = int(std::ceil(std::log2(double(extent) / 255.0)));
    while (std::ldexp(255.0, e) < double(extent)) e++;
    return std::max(e, -126);
}

// Quantise child interval [a, b] in the frame (origin o, scale 2^e) so that
// the decoded interval o + q*2^e, evaluated as the kernel does (fmaf),
// contains it.
void quantise(float o, int e, float a, float b, uint8_t &qa, uint8_t &qb, bool &ok) {
    const float s = std::ldexp(1.0f, e);
    long la = long(std::floor((double(a) - double(o)) / double(s)));
    long lb = long(std::ceil((double(b) - double(o)) / double(s)));
    la = std::max(0L, std::min(255L, la));
    lb = std::max(0L, std::min(255L, lb));
    while (la > 0 && std::fma(float(la), s, o) > a) la--;
    while (lb < 255 && std::fma(float(lb), s, o) < b) lb++;
    ok = ok && std::fma(float(la), s, o) <= a && std::fma(float(lb), s, o) >= b;
    qa = uint8_t(la);
    qb = uint8_t(lb);
}

struct Collapser {
    const ae_bvh_node *bin;  // this mesh's binary nodes
    std::vector<WideNode> &out;
    bool ok = true;
    int max_stack = 0;

    // Children of binary node `i` gathered into up to four: repeatedly open
    // the interior child with the largest surface area.
    uint32_t emit(uint32_t i) {
        std::vector<uint32_t> kids = {uint32_t(bin[i].left), uint32_t(bin[i].right)};
        while (kids.size() < 4) {
            int best = -1;
            float area = -1.0f;
            for (size_t k = 0; k < kids.size(); k++) {
                const ae_bvh_node &c = bin[kids[k]];
                if (c.count > 0) continue;
                const float a = half_area(node_box(c));
                if (a > area) { area = a; best = int(k); }
            }
            if (best < 0) break;
            const uint32_t open = kids[best];
            kids.erase(kids.begin() + best);
            kids.insert(kids.begin() + best, uint32_t(bin[open].right));
            kids.insert(kids.begin() + best, uint32_t(bin[open].left));
        }
        const uint32_t self = uint32_t(out.size());
        out.push_back(WideNode{});
        WideNode q;
        std::memset(&q, 0, sizeof(q));
        Box nb = node_box(bin[i]);
        // Conservative frame: the union of the children.
        Box u = node_box(bin[kids[0]]);
        for (size_t k = 1; k < kids.size(); k++) {
            const Box c = node_box(bin[kids[k]]);
            for (int a = 0; a < 3; a++) { u.lo[a] = std::min(u.lo[a], c.lo[a]); u.hi[a] = std::max(u.hi[a], c.hi[a]); }
        }
        (void)nb;
        q.ox = u.lo[0]; q.oy = u.lo[1]; q.oz = u.lo[2];
        const float org[3] = {q.ox, q.oy, q.oz};
        int ex[3];
        for (int a = 0; a < 3; a++) {
            int e = axis_exponent(u.hi[a] - u.lo[a]);
            // Raise the exponent until the top of the frame is representable.
            for (;;) {
                const float s = std::ldexp(1.0f, e);
                if (std::fma(255.0f, s, org[a]) >= u.hi[a] || e > 127) break;
                e++;
            }
            ex[a] = e;
        }
        q.ex = int8_t(ex[0]); q.ey = int8_t(ex[1]); q.ez = int8_t(ex[2]);
        q.nchild = uint8_t(kids.size());
        for (size_t k = 0; k < kids.size(); k++) {
            const Box c = node_box(bin[kids[k]]);
            for (int a = 0; a < 3; a++) quantise(org[a], ex[a], c.lo[a], c.hi[a], q.lo[a][k], q.hi[a][k], ok);
        }
        for (size_t k = 0; k < kids.size(); k++) {
            const ae_bvh_node &c = bin[kids[k]];
            if (c.count > 0) {
                if (uint32_t(c.count) > kMaxLeafCount || uint32_t(c.left) >= kMaxLeafFirst) ok = false;
                q.child[k] = leaf_ref(uint32_t(c.left) & 0x00ffffffu, uint32_t(c.count) & 0x7fu);
            }
        }
        // Empty slots: an inverted box (lo 255 > hi 0) never hits.
        for (size_t k = kids.size(); k < 4; k++)
            for (int a = 0; a < 3; a++) { q.lo[a][k] = 255; q.hi[a][k] = 0; }
        for (size_t k = 0; k < kids.size(); k++) {
            const ae_bvh_node &c = bin[kids[k]];
            if (c.count <= 0) q.child[k] = emit(kids[k]);
        }
        out[self] = q;
        return self;
    }
};

// Worst-case stack entries of the kernel's loop over this tree: on each
// node the far hit children are pushed (up to nchild - 1).
int stack_need(const std::vector<WideNode> &nodes, uint32_t root) {
    const WideNode &q = nodes[root];
    int best = 0;
    for (int k = 0; k < q.nchild; k++) {
        if (q.child[k] & kLeafBit) continue;
        best = std::max(best, stack_need(nodes, q.child[k]));
    }
    return (q.nchild - 1) + best;
}

// Boxes of a mesh's binary BLAS nodes at depth kSubBoxDepth (leaves above
// that depth count as they are), appended to `out` as six floats each; they
// cover every triangle of the mesh.  Returns how many.
uint32_t mesh_sub_boxes(const ae_bvh_node *bin, std::vector<float> &out) {
    std::vector<uint32_t> level = {0};
    for (int d = 0; d < kSubBoxDepth; d++) {
        std::vector<uint32_t> next;
        for (uint32_t i : level) {
            if (bin[i].count > 0) next.push_back(i);
            else { next.push_back(uint32_t(bin[i].left)); next.push_back(uint32_t(bin[i].right)); }
        }
        level.swap(next);
    }
    for (uint32_t i : level) {
        const ae_bvh_node &n = bin[i];
        const float b[6] = {n.min_x, n.min_y, n.min_z, n.max_x, n.max_y, n.max_z};
        out.insert(out.end(), b, b + 6);
    }
    return uint32_t(level.size());
}

// Binary tree over object boxes with one object per leaf, in ae_bvh_node
// form (a leaf holds its object slot in `left`, count 1): binned SAH over the
// centroids, 16 bins per axis; a median split where the centroids coincide
// or the tree gets deep.
struct ObjectTree {
    const std::vector<Box> &box;
    std::vector<uint32_t> idx;
    std::vector<ae_bvh_node> nodes;

    static float centre(const Box &b, int a) { return 0.5f * (b.lo[a] + b.hi[a]); }

    uint32_t build(uint32_t b, uint32_t e, int depth) {
        const uint32_t self = uint32_t(nodes.size());
        nodes.push_back(ae_bvh_node{});
        Box u = box[idx[b]];
        for (uint32_t i = b + 1; i < e; i++)
            for (int a = 0; a < 3; a++) {
                u.lo[a] = std::min(u.lo[a], box[idx[i]].lo[a]);
                u.hi[a] = std::max(u.hi[a], box[idx[i]].hi[a]);
            }
        ae_bvh_node n;
        std::memset(&n, 0, sizeof(n));
        n.min_x = u.lo[0]; n.min_y = u.lo[1]; n.min_z = u.lo[2];
        n.max_x = u.hi[0]; n.max_y = u.hi[1]; n.max_z = u.hi[2];
        if (e - b == 1) {
            n.left = int32_t(idx[b]);
            n.count = 1;
            nodes[self] = n;
            return self;
        }
        float clo[3] = {1e30f, 1e30f, 1e30f}, chi[3] = {-1e30f, -1e30f, -1e30f};
        for (uint32_t i = b; i < e; i++)
            for (int a = 0; a < 3; a++) {
                clo[a] = std::min(clo[a], centre(box[idx[i]], a));
                chi[a] = std::max(chi[a], centre(box[idx[i]], a));
            }
        constexpr int kBins = 16;
        int axis = -1, split = 0;
        double best = 1e300;
        for (int a = 0; a < 3 && depth < 48; a++) {
            const float ext = chi[a] - clo[a];
            if (!(ext > 0.0f)) continue;
            uint32_t cnt[kBins] = {};
            Box bb[kBins];
            for (int k = 0; k < kBins; k++)
                for (int j = 0; j < 3; j++) { bb[k].lo[j] = 1e30f; bb[k].hi[j] = -1e30f; }
            for (uint32_t i = b; i < e; i++) {
                const Box &x = box[idx[i]];
                const int k = std::min(kBins - 1, int((centre(x, a) - clo[a]) / ext * kBins));
                cnt[k]++;
                for (int j = 0; j < 3; j++) { bb[k].lo[j] = std::min(bb[k].lo[j], x.lo[j]); bb[k].hi[j] = std::max(bb[k].hi[j], x.hi[j]); }
            }
            double right_area[kBins];
            uint32_t right_cnt[kBins];
            Box acc = bb[kBins - 1];
            uint32_t rc = 0;
            for (int k = kBins - 1; k >= 1; k--) {
                if (k < kBins - 1)
                    for (int j = 0; j < 3; j++) { acc.lo[j] = std::min(acc.lo[j], bb[k].lo[j]); acc.hi[j] = std::max(acc.hi[j], bb[k].hi[j]); }
                rc += cnt[k];
                right_area[k] = rc ? half_area(acc) : 0.0;
                right_cnt[k] = rc;
            }
            Box lacc = bb[0];
            uint32_t lc = 0;
            for (int k = 1; k < kBins; k++) {
                if (k > 1)
                    for (int j = 0; j < 3; j++) { lacc.lo[j] = std::min(lacc.lo[j], bb[k - 1].lo[j]); lacc.hi[j] = std::max(lacc.hi[j], bb[k - 1].hi[j]); }
                lc += cnt[k - 1];
                if (!lc || !right_cnt[k]) continue;
                const double cost = double(lc) * half_area(lacc) + double(right_cnt[k]) * right_area[k];
                if (cost < best) { best = cost; axis = a; split = k; }
            }
        }
        uint32_t m = b;
        if (axis >= 0) {
            const float ext = chi[axis] - clo[axis];
            m = uint32_t(std::partition(idx.begin() + b, idx.begin() + e, [&](uint32_t o) {
                            return std::min(kBins - 1, int((centre(box[o], axis) - clo[axis]) / ext * kBins)) < split;
                        }) - idx.begin());
        }
        if (m == b || m == e) {
            int a = 0;
            for (int j = 1; j < 3; j++) if (chi[j] - clo[j] > chi[a] - clo[a]) a = j;
            m = (b + e) / 2;
            std::nth_element(idx.begin() + b, idx.begin() + m, idx.begin() + e,
                             [&](uint32_t x, uint32_t y) { return centre(box[x], a) < centre(box[y], a); });
        }
        const uint32_t l = build(b, m, depth + 1), r = build(m, e, depth + 1);
        n.left = int32_t(l);
        n.right = int32_t(r);
        n.count = 0;
        nodes[self] = n;
        return self;
    }
};

}  // namespace

// The 4-wide quantised BVH of one mesh from its binary BLAS (mesh-relative
// node links, `tri_count` triangles).  Node indices in `out` start at 0; the
// root is returned in `root` (a node index, or a leaf ref for a one-leaf
// mesh).  Checks, before anything reaches a device: every link stays inside
// the tree, every leaf inside the mesh's triangles, every quantised box
// contains its exact box, and the traversal stack bound.
bool build_qbvh(const ae_bvh_node *bin, uint32_t n_bin, uint32_t tri_count, std::vector<WideNode> &out, uint32_t &root,
                int &stack, std::string &err) {
    out.clear();
    stack = 0;
    if (n_bin == 0) { err = "empty BLAS"; return false; }
    // The binary tree itself: links in range, acyclic, leaves in range.
    {
        std::vector<uint8_t> seen(n_bin, 0);
        std::vector<uint32_t> todo = {0};
        while (!todo.empty()) {
            const uint32_t i = todo.back();
            todo.pop_back();
            if (i >= n_bin || seen[i]++) { err = "binary BLAS link out of range or repeated"; return false; }
            const ae_bvh_node &n = bin[i];
            if (n.count > 0) {
                if (n.left < 0 || uint64_t(n.left) + uint64_t(n.count) > tri_count) { err = "leaf outside the mesh"; return false; }
                if (uint32_t(n.count) > kMaxLeafCount || uint32_t(n.left) >= kMaxLeafFirst) {
                    err = "leaf beyond the packed reference limits";
                    return false;
                }
            } else {
                if (n.left < 0 || n.right < 0) { err = "negative link"; return false; }
                todo.push_back(uint32_t(n.left));
                todo.push_back(uint32_t(n.right));
            }
        }
    }
    if (bin[0].count > 0) {
        root = leaf_ref(uint32_t(bin[0].left), uint32_t(bin[0].count));
        stack = 0;
        return true;
    }
    Collapser col{bin, out};
    root = col.emit(0);
    if (!col.ok) { err = "a child box cannot be quantised conservatively"; return false; }
    // Final structural check of what the kernel will follow.
    for (size_t i = 0; i < out.size(); i++) {
        const WideNode &q = out[i];
        if (q.nchild < 2 || q.nchild > 4) { err = "node child count"; return false; }
        for (int k = 0; k < q.nchild; k++) {
            const uint32_t r = q.child[k];
            if (r & kLeafBit) {
                if (leaf_count(r) == 0 || uint64_t(leaf_first(r)) + leaf_count(r) > tri_count) { err = "leaf ref"; return false; }
            } else if (r >= out.size()) {
                err = "node ref";
                return false;
            }
        }
    }
    stack = stack_need(out, root);
    if (stack + 1 > kFastStack) { err = "tree needs more stack than the kernel holds"; return false; }
    return true;
}

// ---------------------------------------------------------------------------
// Instance-level tree
// ---------------------------------------------------------------------------

// Conservative world box of every object, one warp per object: a mesh
// instance's sub-boxes (its BLAS nodes at depth kSubBoxDepth) with each
// corner through the instance transform in double precision, the extremes
// rounded outward to float; an analytic object's packed box.  Both are
// widened by `margin` on every side, which covers the rounding of the
// kernels' ToLocal and triangle arithmetic for rays that start within the
// scene's coordinate range (the margin is 2^-14 of it).
__global__ void k_object_boxes(const uint4 *__restrict__ meta, const FastInst *__restrict__ inst,
                               const float *__restrict__ sub, const uint2 *__restrict__ sub_refs,
                               const float *__restrict__ static_box, uint32_t n,
                               float margin, float *__restrict__ out) {
    const uint32_t slot = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (slot >= n) return;  // whole warps
    const uint4 m = meta[slot];
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    if ((m.x & 0xff) == AE_SHAPE_MESH) {
        const FastInst I = inst[m.y];
        const double s = (I.scale != 0.0f && I.scale != 1.0f) ? double(I.scale) : 1.0;
        const double qx = I.qx, qy = I.qy, qz = I.qz, qw = I.qw;
        const uint2 sr = sub_refs[I.sub];
        const uint32_t first = sr.x, cnt = sr.y;
        for (uint32_t j = lane; j < cnt * 8u; j += 32) {
            const float *x = sub + 6 * size_t(first + j / 8);
            const uint32_t k = j & 7u;
            const double v0 = double(k & 1u ? x[3] : x[0]) * s, v1 = double(k & 2u ? x[4] : x[1]) * s,
                         v2 = double(k & 4u ? x[5] : x[2]) * s;
            const double t0 = 2.0 * (qy * v2 - qz * v1), t1 = 2.0 * (qz * v0 - qx * v2), t2 = 2.0 * (qx * v1 - qy * v0);
            const double w[3] = {v0 + qw * t0 + (qy * t2 - qz * t1) + double(I.px),
                                 v1 + qw * t1 + (qz * t0 - qx * t2) + double(I.py),
                                 v2 + qw * t2 + (qx * t1 - qy * t0) + double(I.pz)};
            for (int a = 0; a < 3; a++) { lo[a] = fmin(lo[a], w[a]); hi[a] = fmax(hi[a], w[a]); }
        }
        for (int off = 16; off > 0; off >>= 1)
            for (int a = 0; a < 3; a++) {
                lo[a] = fmin(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], off));
                hi[a] = fmax(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], off));
            }
    } else {
        const float *x = static_box + 6 * size_t(slot);
        for (int a = 0; a < 3; a++) { lo[a] = x[a]; hi[a] = x[3 + a]; }
    }
    if (lane == 0) {
        float *o = out + 6 * size_t(slot);
        for (int a = 0; a < 3; a++) {
            o[a] = __fsub_rd(__double2float_rd(lo[a]), margin);
            o[3 + a] = __fadd_ru(__double2float_ru(hi[a]), margin);
        }
    }
}

// One level of the instance tree's bottom-up refresh (levels deepest first):
// a node's float box is the union of its children's (objects' boxes for leaf
// children), and its children are re-quantised in the node's new frame.  A
// child whose box is empty or not finite becomes an unused slot.  Sets *bad
// when a box cannot be quantised conservatively.
__device__ void instance_tree_node(QNode *__restrict__ nodes, float *nbox, const float *__restrict__ obj_box, int32_t ni,
                                   uint32_t *bad) {
    QNode q = nodes[ni];
    int n = 0;
    while (n < 4 && q.child[n] != kNoChild) n++;
    float cb[4][6], u[6];
    bool cv[4];
    for (int c = 0; c < 4; c++) {
        cv[c] = false;
        if (c >= n) continue;
        const uint32_t ref = q.child[c];
        const float *x = (ref & kLeafBit) ? obj_box + 6 * size_t(leaf_first(ref)) : nbox + 6 * size_t(ref);
        bool ok = true;
        for (int a = 0; a < 6; a++) { cb[c][a] = x[a]; ok = ok && isfinite(x[a]); }
        for (int a = 0; a < 3; a++) ok = ok && cb[c][a] <= cb[c][3 + a];
        cv[c] = ok;
    }
    if (!quantise_node(q, n, cb, cv, u)) atomicExch(bad, 1u);
    nodes[ni] = q;
    float *o = nbox + 6 * size_t(ni);
    for (int a = 0; a < 6; a++) o[a] = u[a];
}
__global__ void k_instance_tree_level(QNode *nodes, float *nbox, const float *obj_box, const int32_t *level, int32_t count,
                                      uint32_t *bad) {
    const int32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < count) instance_tree_node(nodes, nbox, obj_box, level[k], bad);
}
// All levels by one block (as k_refit_levels, refit.cu).
__global__ void __launch_bounds__(256) k_instance_tree_levels(QNode *nodes, float *nbox, const float *obj_box,
                                                              const int32_t *order, const int32_t *start, int32_t levels,
                                                              uint32_t *bad) {
    for (int32_t l = 0; l < levels; l++) {
        for (int32_t k = start[l] + int32_t(threadIdx.x); k < start[l + 1]; k += int32_t(blockDim.x))
            instance_tree_node(nodes, nbox, obj_box, order[k], bad);
        __syncthreads();
    }
}

// Instance records after a refit: the transforms of the uploaded instances.
__global__ void k_move_instances(FastInst *__restrict__ inst, const ae_instance *__restrict__ from, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const ae_instance m = from[i];
    FastInst f = inst[i];
    f.px = m.px; f.py = m.py; f.pz = m.pz; f.scale = m.scale;
    f.qx = m.qx; f.qy = m.qy; f.qz = m.qz; f.qw = m.qw;
    f.inv_scale = m.scale != 0.0f && m.scale != 1.0f ? AE_DIV(1.0f, m.scale) : 1.0f;
    inst[i] = f;
}

// Per object, the intersection of the reference TLAS boxes above it, leaf to
// root (exact_trace.cuh); an object in no reachable leaf gets an empty box.
__global__ void k_object_chain(const uint4 *__restrict__ meta, const ae_bvh_node *__restrict__ tlas,
                               const int32_t *__restrict__ parent, uint32_t n, float4 *__restrict__ out) {
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const float inf = __int_as_float(0x7f800000);
    float4 lo = make_float4(-inf, -inf, -inf, 0.0f), hi = make_float4(inf, inf, inf, 0.0f);
    int32_t i = int32_t(meta[s].w);
    if (i < 0) lo.x = inf;
    for (; i >= 0; i = parent[i]) {
        const NodeBox b = load_node(tlas, uint32_t(i));
        lo.x = fmaxf(lo.x, b.lo.x); lo.y = fmaxf(lo.y, b.lo.y); lo.z = fmaxf(lo.z, b.lo.z);
        hi.x = fminf(hi.x, b.hi.x); hi.y = fminf(hi.y, b.hi.y); hi.z = fminf(hi.z, b.hi.z);
    }
    out[2 * s] = lo;
    out[2 * s + 1] = hi;
}

// Topology of the instance-level tree for the current objects (host, per
// scene layout): an object tree over host bounds, collapsed 4-wide by the
// BLAS collapser.  The boxes uploaded here are replaced by the device
// refresh.
static int build_instance_tree(Ctx *c, FastScene &F) {
    const uint32_t n = c->n_objects;
    F.n_tnodes = 0;
    F.tlas_stack = 0;
    F.troot = kEmptyTlas;
    F.static_range = 0.0f;
    if (n == 0) return AE_OK;
    if (n >= kMaxLeafFirst) return c->fail(AE_ERR_LAYOUT, "%u objects: the instance tree addresses at most %u", n, kMaxLeafFirst);
    // Mesh objects' boxes by the refresh kernel (no margin): 256 sub-boxes of
    // eight corners an instance took the host 10 us each (1,024 instances: prepare
    // 14.6 -> 3.8 ms).
    if (F.obj_box.reserve(size_t(n) * 6) || F.static_box.reserve(size_t(n) * 6)) return c->fail(AE_ERR_OOM, "instance tree");
    k_object_boxes<<<(n * 32 + 255) / 256, 256, 0, c->stream>>>(F.obj_meta.ptr, F.inst.ptr, F.sub_boxes.ptr, F.sub_refs.ptr,
                                                                 F.static_box.ptr, n, 0.0f, F.obj_box.ptr);
    std::vector<float> world(size_t(n) * 6);
    int rc;
    if ((rc = c->cuda(cudaGetLastError(), "object boxes")) ||
        (rc = c->cuda(cudaMemcpyAsync(world.data(), F.obj_box.ptr, world.size() * sizeof(float), cudaMemcpyDeviceToHost,
                                      c->stream), "object boxes")) ||
        (rc = c->cuda(cudaStreamSynchronize(c->stream), "object boxes")))
        return rc;
    std::vector<Box> boxes(n);
    std::vector<float> stat(size_t(n) * 6, 0.0f);
    for (uint32_t s = 0; s < n; s++) {
        const ae_object &o = c->host_objects[s];
        if (o.shapeType == AE_SHAPE_MESH) {
            std::memcpy(&boxes[s], &world[6 * size_t(s)], 24);
        } else {
            const ae_aabb b = analytic_box(o);
            boxes[s] = Box{{b.min_x, b.min_y, b.min_z}, {b.max_x, b.max_y, b.max_z}};
            std::memcpy(&stat[6 * size_t(s)], &b, 24);
            // One object at infinity would take the margin of all boxes with it.
            for (int a = 0; a < 3; a++)
                for (const float x : {std::fabs(boxes[s].lo[a]), std::fabs(boxes[s].hi[a])})
                    if (std::isfinite(x)) F.static_range = std::max(F.static_range, x);
        }
    }
    // For the exact walks' widening: the spheres (a radius that is no positive
    // number leaves no finite bound) and the shape factor of the planar objects
    // that the reference test can accept.
    for (double &x : F.sphere) x = 0.0;
    F.planar_factor = 1.0f;
    F.odd_boxes = false;
    for (uint32_t s = 0; s < n; s++) {
        const ae_object &o = c->host_objects[s];
        // The reference walk hits a box of negative half extents, and objects
        // whose NaN passes its slab tests; neither has a box in the tree.  The
        // walks reduce a yaw in binary32, to 2^-24 of the angle: up to 100
        // radians a tenth of the boxes' margin.  (Meshes: plain_transforms.)
        if (o.shapeType != AE_SHAPE_MESH && !box_within(boxes[s], kPlainReach)) F.odd_boxes = true;
        // The object tree's buckets and the collapse need numbers; where such an
        // object lies in the tree does not matter.
        if (!box_within(boxes[s], 1e30f)) boxes[s] = Box{};
        if (o.shapeType == AE_SHAPE_BOX && !(std::fabs(o.rotation) < 100.0f)) F.odd_boxes = true;
        if (o.shapeType == AE_SHAPE_SPHERE) {
            const double r = o.radius > 0.0f ? double(o.radius) : 0.0;
            const double q = std::sqrt(double(o.x) * o.x + double(o.y) * o.y + double(o.z) * o.z) + r;
            const double bound[3] = {1.0 / r, q / r, q * q / r};
            for (int k = 0; k < 3; k++)
                if (!(bound[k] <= F.sphere[k])) F.sphere[k] = bound[k];  // a NaN too
        }
        if (o.shapeType != AE_SHAPE_QUAD && o.shapeType != AE_SHAPE_TRIANGLE) continue;
        const f3 u = mk(o.u_x, o.u_y, o.u_z), v = mk(o.v_x, o.v_y, o.v_z), nn = cross(u, v);
        const float n2 = dot(nn, nn);
        if (n2 < 1e-8f) continue;
        const double f = std::sqrt(double(dot(u, u))) * std::sqrt(double(dot(v, v))) / std::sqrt(double(n2));
        F.planar_factor = f < 1e30 ? std::max(F.planar_factor, float(f)) : 3.402823466e38f;
    }
    ObjectTree T{boxes, {}, {}};
    T.idx.resize(n);
    for (uint32_t s = 0; s < n; s++) T.idx[s] = s;
    T.nodes.reserve(2 * size_t(n));
    T.build(0, n, 0);
    std::vector<WideNode> out;
    uint32_t root;
    if (T.nodes[0].count > 0) {
        root = leaf_ref(uint32_t(T.nodes[0].left), 1);
    } else {
        Collapser col{T.nodes.data(), out};
        root = col.emit(0);
        F.tlas_stack = stack_need(out, root);
        if (F.tlas_stack > kTlas4Stack)
            return c->fail(AE_ERR_LAYOUT, "instance tree needs %d stack entries (> %d)", F.tlas_stack, kTlas4Stack);
    }
    // Nodes by depth, deepest first, for the bottom-up refresh.
    std::vector<int32_t> depth(out.size(), 0), order;
    int maxd = 0;
    for (size_t i = 0; i < out.size(); i++)
        for (int k = 0; k < out[i].nchild; k++)
            if (!(out[i].child[k] & kLeafBit)) {
                depth[out[i].child[k]] = depth[i] + 1;
                maxd = std::max(maxd, depth[i] + 1);
            }
    F.tlevel_start.assign(1, 0);
    for (int d = maxd; d >= 0 && !out.empty(); d--) {
        for (size_t i = 0; i < out.size(); i++)
            if (depth[i] == d) order.push_back(int32_t(i));
        F.tlevel_start.push_back(int32_t(order.size()));
    }
    const size_t nn = std::max<size_t>(out.size(), 1);
    if (F.tnodes.reserve(nn) || F.tbox.reserve(nn * 6) || F.tlevels.reserve(std::max<size_t>(order.size(), 1)) ||
        F.tflag.reserve(1) ||
        F.tlevel_start_dev.reserve(F.tlevel_start.size()))
        return c->fail(AE_ERR_OOM, "instance tree");
    // Links and child counts; the refresh writes frames and planes.
    std::vector<QNode> dev(out.size(), QNode{});
    for (size_t i = 0; i < out.size(); i++) {
        for (int k = 0; k < 4; k++) {
            dev[i].plane[k] = make_uint2(0u, kPlaneUnused);
            dev[i].child[k] = k < out[i].nchild ? out[i].child[k] : kNoChild;
        }
    }
    if (!out.empty() &&
        ((rc = c->cuda(cudaMemcpyAsync(F.tnodes.ptr, dev.data(), dev.size() * sizeof(QNode), cudaMemcpyHostToDevice,
                                       c->stream), "upload instance tree")) ||
         (rc = c->cuda(cudaMemcpyAsync(F.tlevels.ptr, order.data(), order.size() * sizeof(int32_t),
                                       cudaMemcpyHostToDevice, c->stream), "upload instance tree levels")) ||
         (rc = c->cuda(cudaMemcpyAsync(F.tlevel_start_dev.ptr, F.tlevel_start.data(), F.tlevel_start.size() * sizeof(int32_t),
                                       cudaMemcpyHostToDevice, c->stream), "upload instance tree levels"))))
        return rc;
    if ((rc = c->cuda(cudaMemcpyAsync(F.static_box.ptr, stat.data(), stat.size() * sizeof(float), cudaMemcpyHostToDevice,
                                      c->stream), "upload object boxes")))
        return rc;
    // The host copies must outlive the asynchronous copies.
    if ((rc = c->cuda(cudaStreamSynchronize(c->stream), "instance tree"))) return rc;
    F.n_tnodes = uint32_t(out.size());
    F.troot = root;
    return AE_OK;
}

// Device refresh of the instance tree's boxes from the current instance
// records (after every upload or refit).
static int refresh_instance_tree(Ctx *c, FastScene &F) {
    // Coordinate range of the scene for the margin of the object boxes.
    float range = 1.0f;
    for (uint32_t s = 0; s < c->n_objects; s++) {
        const ae_object &o = c->host_objects[s];
        if (o.shapeType == AE_SHAPE_MESH) {
            const ae_instance &m = c->host_instances[o.instanceIndex];
            const float sc = (m.scale != 0.0f && m.scale != 1.0f) ? std::fabs(m.scale) : 1.0f;
            const float r = std::max(std::fabs(m.px), std::max(std::fabs(m.py), std::fabs(m.pz))) +
                            1.75f * sc * F.inst_radius[o.instanceIndex];
            if (std::isfinite(r)) range = std::max(range, r);
        }
    }
    range = std::max(range, F.static_range);
    F.range = range;
    const float margin = std::ldexp(range, -14);
    const uint32_t n = c->n_objects;
    int rc;
    if (n == 0) return AE_OK;
    k_object_chain<<<(n + 127) / 128, 128, 0, c->stream>>>(F.obj_meta.ptr, c->tlas.ptr, F.tlas_parent.ptr, n,
                                                          F.obj_chain.ptr);
    if (F.n_tnodes == 0) return c->cuda(cudaGetLastError(), "instance tree refresh");
    if ((rc = c->cuda(cudaMemsetAsync(F.tflag.ptr, 0, sizeof(uint32_t), c->stream), "instance tree flag"))) return rc;
    k_object_boxes<<<(n * 32 + 255) / 256, 256, 0, c->stream>>>(F.obj_meta.ptr, F.inst.ptr, F.sub_boxes.ptr, F.sub_refs.ptr,
                                                                 F.static_box.ptr, n, margin, F.obj_box.ptr);
    const bool one_block = F.n_tnodes <= 1024;
    if (one_block)
        k_instance_tree_levels<<<1, 256, 0, c->stream>>>(F.tnodes.ptr, F.tbox.ptr, F.obj_box.ptr, F.tlevels.ptr,
                                                         F.tlevel_start_dev.ptr, int32_t(F.tlevel_start.size()) - 1,
                                                         F.tflag.ptr);
    for (size_t l = 0; !one_block && l + 1 < F.tlevel_start.size(); l++) {
        const int32_t cnt = F.tlevel_start[l + 1] - F.tlevel_start[l];
        if (cnt <= 0) continue;
        k_instance_tree_level<<<(cnt + 127) / 128, 128, 0, c->stream>>>(F.tnodes.ptr, F.tbox.ptr, F.obj_box.ptr,
                                                                       F.tlevels.ptr + F.tlevel_start[l], cnt, F.tflag.ptr);
    }
    return c->cuda(cudaGetLastError(), "instance tree refresh");
}

// The reference walk's answer to a ray whose direction is NaN on every axis.
// Its slab tests drop NaN distances, so it enters the first leaf it reaches
// (right children first), where every comparison against a NaN t fails and so
// accepts: each object that can be hit replaces the one before.  The far bound
// is then NaN, which fails every further slab test, a mesh's root included.
// In a mesh, the first leaf with a triangle that is not degenerate decides,
// by its last such triangle.  The watertight test refuses a NaN t, boxes
// refuse a NaN interval; spheres and planar objects accept.
static void nan_answers(const Ctx *c, FastScene &F) {
    const uint2 none = make_uint2(AE_MISS, AE_MISS);
    auto mesh_triangle = [&](const ae_instance &m) {
        uint32_t found = AE_MISS;
        std::vector<int32_t> todo = {0};
        while (!todo.empty() && found == AE_MISS) {
            const ae_bvh_node &n = c->host_blas[m.blasBase + todo.back()];
            todo.pop_back();
            if (n.count <= 0) {
                todo.push_back(n.left);
                todo.push_back(n.right);
                continue;
            }
            for (int32_t k = 0; k < n.count; k++) {
                f3 p[3];
                for (int v = 0; v < 3; v++) {
                    const ae_vertex &x = c->host_vertices[m.vertexBase + c->host_indices[m.indexBase + 3 * (n.left + k) + v]];
                    p[v] = mk(x.px, x.py, x.pz);
                }
                const f3 nn = cross(p[1] - p[0], p[2] - p[0]);
                if (!(dot(nn, nn) < 1e-12f)) found = uint32_t(n.left + k);
            }
        }
        return found;
    };
    for (int wt = 0; wt < 2; wt++) {
        uint2 hit = none;
        std::vector<int32_t> todo;
        if (c->n_nodes) todo.push_back(0);
        while (!todo.empty() && hit.x == AE_MISS) {
            const ae_bvh_node &n = c->host_tlas[todo.back()];
            todo.pop_back();
            if (n.count <= 0) {
                todo.push_back(n.left);
                todo.push_back(n.right);
                continue;
            }
            for (int32_t k = 0; k < n.count; k++) {
                const uint32_t slot = uint32_t(n.left + k);
                const ae_object &o = c->host_objects[slot];
                if (o.shapeType == AE_SHAPE_MESH) {
                    const uint32_t t = wt || hit.x != AE_MISS ? AE_MISS : mesh_triangle(c->host_instances[o.instanceIndex]);
                    if (t != AE_MISS) hit = make_uint2(slot, t);
                } else if (o.shapeType == AE_SHAPE_SPHERE) {
                    hit = make_uint2(slot, AE_MISS);
                } else if (o.shapeType != AE_SHAPE_BOX) {
                    const f3 nn = cross(mk(o.u_x, o.u_y, o.u_z), mk(o.v_x, o.v_y, o.v_z));
                    if (!(dot(nn, nn) < 1e-8f)) hit = make_uint2(slot, AE_MISS);
                }
            }
        }
        (wt ? F.nan_wt : F.nan_ref) = hit;
    }
}

int prepare_fast(Ctx *c) {
    // Not ready until this call accepts the current scene: every early
    // return below leaves the optimised structures unusable.
    c->fast_ready = false;
    if (c->fast && c->fast->geometry_key == c->geometry_version && c->fast->scene_key == c->scene_version &&
        !c->fast->geometry_dirty && !c->fast->has_volumes) {
        // Built for exactly this scene: nothing to look at again.
        c->fast_ready = true;
        c->fast_accepted = c->scene_version;
        return AE_OK;
    }
    if (!c->geometry_uploaded || !c->scene_uploaded) return c->fail(AE_ERR_STATE, "prepare before uploads");
    if (!c->fast) c->fast = new (std::nothrow) FastScene();
    if (!c->fast) return c->fail(AE_ERR_OOM, "fast scene");
    FastScene &F = *c->fast;
    if (F.geometry_key != c->geometry_version) {
        // The host's and the device's builders follow the instances' ranges and
        // trees, which a geometry upload after the scene's may have changed.
        if (const int bad = check_scene_meshes(c)) return bad;
        // New geometry arrays: every mesh is converted again (the device
        // buffers are reused).
        F.mesh_roots.clear();
        F.n_tris = 0;
        F.mesh_sub.clear();
        F.host_sub.clear();
        F.max_stack = 0;
        F.mesh_range = 0.0f;
        F.shade16_tris = 0;
        F.geometry_key = c->geometry_version;
        F.geometry_dirty = true;
    }
    // Only transforms moved since the last build (ae_refit_instances keeps the
    // meshes and the layout): the records are on the device already, and their
    // transforms come from the instances that the refit uploaded.
    const bool moved = !F.geometry_dirty && F.tlas_key == c->scene_version_layout && F.sub_key == c->geometry_version &&
                       F.inst_radius.size() == c->n_instances;
    // Geometry-derived part: rebuilt when new meshes appear.
    bool rebuilt = false;
    for (uint32_t i = 0; !moved && i < c->n_instances; i++) {
        const ae_instance &m = c->host_instances[i];
        const auto key = std::make_tuple(m.vertexBase, m.indexBase, m.triangleCount, m.blasBase);
        if (F.mesh_roots.count(key)) continue;
        // The root reference is filled in by the build; triangle records are
        // numbered in the order in which the meshes are met.
        if (m.triangleCount > 0xffffffffu - F.n_tris) return c->fail(AE_ERR_LAYOUT, "more than 2^32 triangles");
        F.mesh_roots[key] = std::make_pair(0u, F.n_tris);
        F.n_tris += m.triangleCount;
        FastScene::MeshSub ms;
        ms.index = uint32_t(F.mesh_sub.size());
        ms.first = uint32_t(F.host_sub.size() / 6);
        ms.count = mesh_sub_boxes(c->host_blas.data() + m.blasBase, F.host_sub);
        ms.radius = 0.0f;
        for (size_t k = size_t(ms.first) * 6; k < F.host_sub.size(); k++) ms.radius = std::max(ms.radius, std::fabs(F.host_sub[k]));
        F.mesh_range = std::max(F.mesh_range, ms.radius);
        F.mesh_sub[key] = ms;
        F.geometry_dirty = true;
    }
    int rc;
    if (F.geometry_dirty) {
        rebuilt = true;
        if ((rc = build_mesh_structures(c, F))) return rc;
        if (F.sub_boxes.reserve(std::max<size_t>(F.host_sub.size(), 1))) return c->fail(AE_ERR_OOM, "mesh sub-boxes");
        if (!F.host_sub.empty() &&
            (rc = c->cuda(cudaMemcpyAsync(F.sub_boxes.ptr, F.host_sub.data(), F.host_sub.size() * sizeof(float),
                                          cudaMemcpyHostToDevice, c->stream), "upload mesh sub-boxes")))
            return rc;
        std::vector<uint2> sub_refs(std::max<size_t>(F.mesh_sub.size(), 1), make_uint2(0u, 0u));
        for (const auto &kv : F.mesh_sub) sub_refs[kv.second.index] = make_uint2(kv.second.first, kv.second.count);
        if (F.sub_refs.reserve(sub_refs.size())) return c->fail(AE_ERR_OOM, "mesh sub-boxes");
        if ((rc = c->cuda(cudaMemcpyAsync(F.sub_refs.ptr, sub_refs.data(), sub_refs.size() * sizeof(uint2),
                                          cudaMemcpyHostToDevice, c->stream), "upload mesh sub-boxes")) ||
            (rc = c->cuda(cudaStreamSynchronize(c->stream), "mesh sub-boxes")))
            return rc;
        F.geometry_dirty = false;
    }
    // Scene-derived part: instances and object metadata, per upload.
    if (moved && F.scene_key != c->scene_version && c->n_instances)
        k_move_instances<<<(c->n_instances + 127) / 128, 128, 0, c->stream>>>(F.inst.ptr, c->instances.ptr, c->n_instances);
    if (!moved && (F.scene_key != c->scene_version || rebuilt)) {
        F.inst_radius.assign(c->n_instances, 0.0f);
        std::vector<FastInst> fi(std::max<uint32_t>(c->n_instances, 1));
        for (uint32_t i = 0; i < c->n_instances; i++) {
            const ae_instance &m = c->host_instances[i];
            const auto &rt = F.mesh_roots[std::make_tuple(m.vertexBase, m.indexBase, m.triangleCount, m.blasBase)];
            FastInst &f = fi[i];
            f.px = m.px; f.py = m.py; f.pz = m.pz; f.scale = m.scale;
            f.qx = m.qx; f.qy = m.qy; f.qz = m.qz; f.qw = m.qw;
            f.root = rt.first;
            f.tri_base = rt.second;
            const FastScene::MeshSub &ms = F.mesh_sub.at(std::make_tuple(m.vertexBase, m.indexBase, m.triangleCount, m.blasBase));
            f.inv_scale = m.scale != 0.0f && m.scale != 1.0f ? 1.0f / m.scale : 1.0f;
            f.sub = ms.index;
            F.inst_radius[i] = ms.radius;
        }
        // Each object's rank comes from the reference TLAS leaf that holds it.
        std::vector<uint32_t> leaf_first_of(std::max<uint32_t>(c->n_objects, 1), 0u);
        for (const ae_bvh_node &nd : c->host_tlas)
            if (nd.count > 0)
                for (int32_t k = 0; k < nd.count; k++)
                    if (uint32_t(nd.left + k) < c->n_objects) leaf_first_of[nd.left + k] = uint32_t(nd.left);
        // Reachable leaf of each object and the nodes' parents.
        std::vector<int32_t> parent(std::max<uint32_t>(c->n_nodes, 1), -1), leaf_of(std::max<uint32_t>(c->n_objects, 1), -1);
        std::vector<int32_t> todo;
        if (c->n_nodes) todo.push_back(0);
        while (!todo.empty()) {
            const int32_t i = todo.back();
            todo.pop_back();
            const ae_bvh_node &nd = c->host_tlas[i];
            if (nd.count > 0) {
                for (int32_t k = 0; k < nd.count; k++) leaf_of[nd.left + k] = i;
                continue;
            }
            parent[nd.left] = parent[nd.right] = i;
            todo.push_back(nd.left);
            todo.push_back(nd.right);
        }
        std::vector<uint4> meta(std::max<uint32_t>(c->n_objects, 1));
        F.has_volumes = false;
        for (uint32_t s = 0; s < c->n_objects; s++) {
            const ae_object &o = c->host_objects[s];
            meta[s] = make_uint4(o.shapeType | (o.colorType << 8), o.instanceIndex, leaf_first_of[s], uint32_t(leaf_of[s]));
            if (o.colorType == AE_MAT_ISOTROPIC) F.has_volumes = true;
        }
        if (F.inst.reserve(fi.size()) || F.obj_meta.reserve(meta.size()) || F.tlas_parent.reserve(parent.size()) ||
            F.obj_chain.reserve(2 * meta.size()))
            return c->fail(AE_ERR_OOM, "fast scene");
        if ((rc = c->cuda(cudaMemcpyAsync(F.tlas_parent.ptr, parent.data(), parent.size() * sizeof(int32_t),
                                          cudaMemcpyHostToDevice, c->stream), "upload TLAS parents")))
            return rc;
        if ((rc = c->cuda(cudaMemcpyAsync(F.inst.ptr, fi.data(), fi.size() * sizeof(FastInst), cudaMemcpyHostToDevice,
                                          c->stream), "upload instances")))
            return rc;
        if ((rc = c->cuda(cudaMemcpyAsync(F.obj_meta.ptr, meta.data(), meta.size() * sizeof(uint4),
                                          cudaMemcpyHostToDevice, c->stream), "upload metadata")))
            return rc;
        if (F.tlas_key != c->scene_version_layout || F.sub_key != c->geometry_version) {
            F.tlas_key = ~0ull;
            if ((rc = build_instance_tree(c, F))) return rc;
            nan_answers(c, F);
            F.tlas_key = c->scene_version_layout;
            F.sub_key = c->geometry_version;
        }
    }
    if (F.scene_key != c->scene_version || rebuilt) {
        if ((rc = refresh_instance_tree(c, F))) return rc;
        if ((rc = c->cuda(cudaStreamSynchronize(c->stream), "prepare fast"))) return rc;
        if (F.n_tnodes) {
            uint32_t bad = 0;
            if ((rc = c->cuda(cudaMemcpy(&bad, F.tflag.ptr, sizeof(uint32_t), cudaMemcpyDeviceToHost), "instance tree flag")))
                return rc;
            if (bad) return c->fail(AE_ERR_LAYOUT, "instance tree: an object box cannot be quantised conservatively");
        }
        F.scene_key = c->scene_version;
    }
    if (F.has_volumes)
        return c->fail(AE_ERR_STATE, "participating media consume RNG in the reference's visit order; use the plain kernel");
    c->fast_ready = true;
    c->fast_accepted = c->scene_version;
    return AE_OK;
}

// The exact walks' view of the scene (exact_trace.cuh) for a frame or batch of
// `rays` starting rays; off for a call that traces none (a frame that only
// grades its image again) and where the plain walks have to answer: participating
// media (they draw random numbers in visit order), spheres that move within a
// frame (their boxes hold one position), rotations that are not of unit length
// and transforms that are no plain numbers (plain_transforms), objects without
// a box that holds them (odd_boxes), triangles so thin that the widening would
// swallow the scene, uploaded trees whose boxes do not hold their triangles, or
// structures that cannot be built.
//
// Structures that are not current are brought up to date once they would have
// saved the calls made without them (this one included) what they cost, so a
// scene that is asked little never pays, and one that is asked much pays about
// once.  Both sides are times of whole calls on new scenes (means of three):
//
//   prepare, with its allocations and host work, ms: Cornell box 0.37, textured
//   box (11 objects, 1,290 triangles) 0.46, 62,410 triangles in 64 instances
//   1.8, 249,848 in 256 2.5, 523,270 in 200 2.4, 2.1M in 64 2.9, 2.0M in 1,024
//   4.4;
//   saved for each starting ray, ns: compute-only frames 18 (62,410 triangles,
//   depth 4), 54 (249,848, depth 8), 14 (229,894, depth 2), 1.1 (textured box,
//   depth 6), 0.35 (Cornell box, depth 8); hybrid frames, a ray each for
//   G-buffer and resolve, 1.8 (249,848, 4 lights), 33 (2.0M, 16 lights), 0.6
//   (17 objects of 160 triangles); any hit 5.2 (523,270), 3.2 (2.1M).
//
// On a handful of objects with a handful of triangles the reference walk is as
// short and has nothing to verify: any hit 0.072 against 0.090 ms for 200,003
// segments in the Cornell box, hybrid frames of 480x270 216 against 263 us (5
// objects with 160 triangles 245 against 149 us).  AUTO leaves those calls to
// it.  A move refreshes the instance tree alone.
static double saved_ns(const Ctx *c, PlainForm form, bool small) {
    const bool big = c->scene_triangles >= 10000;
    const double depth = double(std::min(c->config.depth, 8u));
    switch (form) {
    case kPlainCompute: return small ? 0.3 : (big ? 5.0 : 0.15) * depth;
    case kPlainHybrid: return big ? 0.4 * (1.0 + double(c->n_lights)) : 0.5;
    default: return big ? 5.0 : 0.5;
    }
}
static double build_ns(const Ctx *c) {
    return 0.5e6 + (c->n_indices >= 30000 ? 1.4e6 : 0.0) + 1800.0 * double(c->n_objects) + 0.13 * double(c->n_indices);
}
ExactView exact_view(Ctx *c, PlainForm form, uint64_t rays) {
    ExactView X;
    std::memset(&X, 0, sizeof(X));
    c->plain_exact = false;
    if (rays == 0 || c->plain_walk == AE_PLAIN_WALK_REFERENCE) return X;
    if (c->scene_has_media || c->scene_has_moving_spheres || !c->scene_plain || c->n_nodes == 0) return X;
    const bool small = c->n_objects < 16 && c->scene_triangles < 128;
    if (small && form != kPlainCompute && c->plain_walk == AE_PLAIN_WALK_AUTO) return X;
    const bool built = c->fast && c->fast->geometry_key == c->geometry_version && !c->fast->geometry_dirty;
    if (!built || c->fast->scene_key != c->scene_version) {
        if (c->plain_walk != AE_PLAIN_WALK_AUTO || c->exact_refused == c->scene_version) return X;
        if (c->plain_scene != c->scene_version) c->plain_scene_ns = 0.0;
        if (c->plain_geometry != c->geometry_version) c->plain_geometry_ns = 0.0;
        c->plain_scene = c->scene_version;
        c->plain_geometry = c->geometry_version;
        const double now = double(rays) * saved_ns(c, form, small);
        c->plain_scene_ns += now;
        c->plain_geometry_ns += now;
        const bool moved = built && c->fast->tlas_key == c->scene_version_layout;
        const double objects = double(c->n_objects), saved = built ? c->plain_scene_ns : c->plain_geometry_ns;
        const double cost = !built ? build_ns(c) : moved ? 1.0e5 + 100.0 * objects : 2.0e5 + 1500.0 * objects;
        if (saved < cost) return X;
        // A build allocates and synchronises, which a stream that is being
        // captured does not allow.
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(c->stream, &capture) != cudaSuccess) cudaGetLastError();
        if (capture != cudaStreamCaptureStatusNone) return X;
    }
    // What the caller asked for is not an optimised form: a failure here is
    // not its failure, and ae_closest_hit_noalloc still wants its own
    // ae_prepare_fast.
    const bool ready = c->fast_ready;
    const uint64_t accepted = c->fast_accepted;
    std::string err = c->err;
    // Another stream of this thread may be under capture, which a global-mode
    // capture would let the allocations break.
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    const int rc = prepare_fast(c);
    cudaThreadExchangeStreamCaptureMode(&mode);
    c->fast_ready = ready;
    c->fast_accepted = accepted;
    c->err.swap(err);
    if (rc) {
        c->exact_refused = c->scene_version;  // not tried again until the scene changes or the caller prepares it
        return X;
    }
    const FastScene &F = *c->fast;
    const float factor = std::max(F.tri_factor, F.planar_factor);
    if (!(factor <= 4096.0f) || F.loose_trees || F.odd_boxes || !(F.mesh_range < kPlainReach)) return X;
    X.V = fast_view(F);
    X.chain = F.obj_chain.ptr;
    X.k = std::ldexp(factor, -17);
    X.world_r = F.range;
    X.mesh_r = F.mesh_range;
    X.max_origin = 3.0e38f;
    if (F.sphere[0] != 0.0) {
        // Origins for which the spheres' widening stays below 2^-8 of the
        // scene; no exact walk where there is none.
        const double a = std::ldexp(F.sphere[0], -19), b = std::ldexp(F.sphere[1], -19), q = std::ldexp(F.sphere[2], -19);
        const double most = (std::sqrt(b * b + a * (std::ldexp(double(F.range), -8) - q)) - b) / a;
        if (!(most > 0.0 && a < 1e30 && b < 1e30)) return X;
        X.sphere_a = float(a);
        X.sphere_b = float(2.0 * b);
        X.sphere_c = float(q);
        X.max_origin = float(std::min(most, 3.0e38));
    }
    X.on = 1;
    c->plain_exact = true;
    return X;
}

void destroy_fast(Ctx *c) {
    delete c->fast;
    c->fast = nullptr;
}

// Closest hit over a ray batch; one thread per ray.  The occupancy bound
// (8 blocks of 128 per SM, so at most 64 registers) was chosen by timing on
// the B200: 1080p camera rays 772 us, against 788 us at 7 and 854 us at 6
// blocks.
template <bool WT>
__global__ void __launch_bounds__(128, 8) k_closest_fast(DevScene S, FastView V, const ae_ray *__restrict__ rays,
                                                      uint32_t n, uint32_t lanes, ae_hit *__restrict__ hits) {
    extern __shared__ uint2 stk[];
    const uint32_t lane = threadIdx.x & 31u, i = (blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32) * lanes + lane;
    if (lane >= lanes || i >= n) return;
    const float4 *rp = reinterpret_cast<const float4 *>(rays + i);
    const float4 r0 = __ldg(rp), r1 = __ldg(rp + 1);
    const Best best = closest_fast<WT>(S, V, mk(r0.x, r0.y, r0.z), mk(r1.x, r1.y, r1.z), r0.w, r1.w, stk,
                                       threadIdx.x, blockDim.x);
    const bool any = best.object != AE_MISS;
    ae_hit out;
    out.t = any ? best.t : 0.0f;
    out.alpha = any ? best.alpha : 0.0f;
    out.beta = any ? best.beta : 0.0f;
    out.object = best.object;
    out.prim = best.prim;
    hits[i] = out;
}

// The optimised walk with its touches counted (outside timed regions): per
// ray set, TLAS nodes, object metadata records, instance records, wide BLAS
// nodes and triangle records fetched, summed in 64-bit.
template <bool WT>
__global__ void __launch_bounds__(128) k_count_fast(DevScene S, FastView V, const ae_ray *__restrict__ rays,
                                                    uint32_t n, unsigned long long *__restrict__ totals) {
    extern __shared__ uint2 stk[];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    Touch T = {0, 0, 0, 0, 0, 0, 0};
    if (i < n) {
        const float4 *rp = reinterpret_cast<const float4 *>(rays + i);
        const float4 r0 = __ldg(rp), r1 = __ldg(rp + 1);
        const Best best = closest_fast<WT>(S, V, mk(r0.x, r0.y, r0.z), mk(r1.x, r1.y, r1.z), r0.w, r1.w, stk,
                                           threadIdx.x, blockDim.x, &T);
        T.winners = best.object != AE_MISS ? 1u : 0u;
    }
    const uint32_t v[6] = {T.tlas, T.objects, T.instances, T.blas, T.tris, T.winners};
    for (int k = 0; k < 6; k++) {
        unsigned long long x = v[k];
        for (int off = 16; off > 0; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
        if ((threadIdx.x & 31) == 0 && x) atomicAdd(totals + k, x);
    }
}

// The same closest hit on the step-wise Walker, for incoherent ray sets
// (bounce rays): a persistent grid where each lane starts its next ray as soon
// as one finishes.  Bit-identical hits.
//
// DYN: rays are handed out in chunks of kWalkChunk consecutive rays per warp
// from a global counter, and the lanes of a warp take theirs from the warp's
// current chunk, so the rays a warp has in flight stay close in the input
// order (neighbouring pixels: neighbouring origins and nodes).  On a
// 1.3M-ray bounce set this took 3.70 -> 3.31 ms; on the current walker, runs
// of 32 rays beat 64 and 128 (1.72 / 1.76 / 1.96 ms).  It keeps every block busy
// to the end of the launch, which suits a launch that has the GPU to itself;
// the smaller launches of the pipelined host-buffer call, which overlap on
// three streams, use the static assignment (lane i: rays i, i + grid size,
// ...), whose blocks retire early and make room for the next launch.
constexpr uint32_t kWalkChunk = 32;
// Eight resident blocks per SM (64 registers): 300,001 pinned host rays 714 -> 696
// us, 1080p bounce rays 841 -> 832 us against seven.
constexpr uint32_t kWalkDynamicMin = (1u << 19) + 1;  // above the host pipeline's largest chunk

template <bool DYN>
__global__ void __launch_bounds__(128, 8) k_closest_walk(DevScene S, FastView V,
                                                                     const ae_ray *__restrict__ rays, uint32_t n,
                                                                     ae_hit *__restrict__ hits, uint32_t *next) {
    extern __shared__ uint2 stk[];
    if (!DYN) {
        const uint32_t warps = gridDim.x * (blockDim.x / 32), lanes = spread_lanes(n, warps);
        const uint32_t stride = warps * lanes;
        uint32_t k = (blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32) * lanes + (threadIdx.x & 31u);
        Walker<false> w;
        WalkStacks<> K;
        bool active = (threadIdx.x & 31u) < lanes && k < n;
        if (active) {
            const ae_ray r = rays[k];
            w.start(V, mk(r.ox, r.oy, r.oz), mk(r.dx, r.dy, r.dz), r.tnear, r.time);
        }
        uint32_t iter = 0;
        for (;;) {
            const uint32_t am = __ballot_sync(0xffffffffu, active);
            if (!am) break;
            // Only the warp's largest phase group steps (warp_pick_group).
            const uint32_t pick = warp_pick_group(active ? w.group() : 0u, active, am, iter);
            if (!active || w.group() != pick || !w.step(S, V, K, stk, threadIdx.x, blockDim.x)) continue;
            const Best &b = w.best;
            const bool any = b.object != AE_MISS;
            ae_hit h;
            h.t = any ? b.t : 0.0f;
            h.alpha = any ? b.alpha : 0.0f;
            h.beta = any ? b.beta : 0.0f;
            h.object = b.object;
            h.prim = b.prim;
            hits[k] = h;
            k += stride;
            active = k < n;
            if (active) {
                const ae_ray r = rays[k];
                w.start(V, mk(r.ox, r.oy, r.oz), mk(r.dx, r.dy, r.dz), r.tnear, r.time);
            }
        }
        return;
    }
    const uint32_t lane = threadIdx.x & 31, below = (1u << lane) - 1u;
    Walker<false> w;
    WalkStacks<> K;
    uint32_t k = 0, cbase = 0, cend = 0;  // cbase/cend: the warp's chunk, the same in every lane
    uint32_t iter = 0;
    bool active = false, need = true, exhausted = false;
    for (;;) {
        // Lanes without a ray take the next ones of the warp's chunk, in lane
        // order; a new chunk is fetched when it runs out.
        uint32_t m = __ballot_sync(0xffffffffu, need);
        while (m && !exhausted) {
            if (cbase >= cend) {
                uint32_t b = 0;
                if (lane == 0) b = atomicAdd(next, kWalkChunk);
                b = __shfl_sync(0xffffffffu, b, 0);
                if (b >= n) {
                    exhausted = true;
                    break;
                }
                cbase = b;
                cend = min(b + kWalkChunk, n);
            }
            const uint32_t take = min(cend - cbase, uint32_t(__popc(m)));
            if (need && uint32_t(__popc(m & below)) < take) {
                k = cbase + __popc(m & below);
                need = false;
                active = true;
                const ae_ray r = rays[k];
                w.start(V, mk(r.ox, r.oy, r.oz), mk(r.dx, r.dy, r.dz), r.tnear, r.time);
            }
            cbase += take;
            m = __ballot_sync(0xffffffffu, need);
        }
        const uint32_t am = __ballot_sync(0xffffffffu, active);
        if (!am) break;
        // Only the warp's largest phase group steps (warp_pick_group): on the
        // 1080p bounce set 3.31 -> 2.70 ms.
        const uint32_t pick = warp_pick_group(w.group(), active, am, iter);
        if (active && w.group() == pick && w.step(S, V, K, stk, threadIdx.x, blockDim.x)) {
            const Best &b = w.best;
            const bool any = b.object != AE_MISS;
            ae_hit h;
            h.t = any ? b.t : 0.0f;
            h.alpha = any ? b.alpha : 0.0f;
            h.beta = any ? b.beta : 0.0f;
            h.object = b.object;
            h.prim = b.prim;
            hits[k] = h;
            active = false;
            need = true;
        }
    }
}

cudaError_t launch_closest_walk(Ctx *c, const ae_ray *rays, uint32_t n, ae_hit *hits, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    FastScene &F = *c->fast;
    FastView V = fast_view(F);
    const int threads = 128;
    const size_t smem = size_t(kSharedStack) * threads * sizeof(uint2);
    // A property of the kernel on this architecture.  Contexts on other threads
    // may get here at the same time: the initialiser runs once and the others
    // wait for it.
    static const int per_sm = [&] {
        int blocks = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_closest_walk<true>, threads, smem) != cudaSuccess)
            cudaGetLastError();
        return std::max(blocks, 1);
    }();
    if (spread_quads(n, uint32_t(c->sms) * 8u * 4u)) return launch_closest_fast(c, rays, n, hits, false, st);
    const uint32_t grid = std::min<uint32_t>(uint32_t(per_sm) * uint32_t(c->sms), (n + 3) / 4);  // at least a ray a warp
    if (n < kWalkDynamicMin) {
        k_closest_walk<false><<<grid, threads, smem, st>>>(c->scene(), V, rays, n, hits, nullptr);
        return cudaGetLastError();
    }
    if (F.walk_next.reserve(FastScene::kWalkCounters)) return cudaErrorMemoryAllocation;
    uint32_t *next = F.walk_next.ptr + (F.walk_pos++ % FastScene::kWalkCounters);
    cudaError_t e = cudaMemsetAsync(next, 0, sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    k_closest_walk<true><<<grid, threads, smem, st>>>(c->scene(), V, rays, n, hits, next);
    return cudaGetLastError();
}

cudaError_t launch_count_fast(Ctx *c, const ae_ray *rays, uint32_t n, bool quant, unsigned long long *totals,
                              cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    FastScene &F = *c->fast;
    FastView V = fast_view(F);
    const int threads = 128;
    const size_t smem = size_t(kSharedStack) * threads * sizeof(uint2);
    if (quant) {
        cudaFuncSetAttribute(k_count_fast<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        k_count_fast<true><<<(n + threads - 1) / threads, threads, smem, st>>>(c->scene(), V, rays, n, totals);
    } else {
        cudaFuncSetAttribute(k_count_fast<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        k_count_fast<false><<<(n + threads - 1) / threads, threads, smem, st>>>(c->scene(), V, rays, n, totals);
    }
    return cudaGetLastError();
}

// Closest hit of a small batch, a quad of lanes a ray (quad_walk.cuh), `quads`
// of them in each warp.
template <bool WT>
__global__ void __launch_bounds__(128) k_closest_quad(DevScene S, FastView V, const ae_ray *__restrict__ rays, uint32_t n,
                                                      uint32_t quads, ae_hit *__restrict__ hits) {
    extern __shared__ uint2 stk[];
    const uint32_t q = (threadIdx.x & 31u) >> 2, i = (blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32) * quads + q;
    if (q >= quads || i >= n) return;
    const float4 *rp = reinterpret_cast<const float4 *>(rays + i);
    const float4 r0 = __ldg(rp), r1 = __ldg(rp + 1);
    const Best best = closest_quad<WT>(S, V, mk(r0.x, r0.y, r0.z), mk(r1.x, r1.y, r1.z), r0.w, r1.w, stk);
    if (threadIdx.x & 3u) return;
    const bool any = best.object != AE_MISS;
    ae_hit h;
    h.t = any ? best.t : 0.0f;
    h.alpha = any ? best.alpha : 0.0f;
    h.beta = any ? best.beta : 0.0f;
    h.object = best.object;
    h.prim = best.prim;
    hits[i] = h;
}

cudaError_t launch_closest_fast(Ctx *c, const ae_ray *rays, uint32_t n, ae_hit *hits, bool quant, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    FastScene &F = *c->fast;
    FastView V = fast_view(F);
    const int threads = 128;
    const size_t smem = size_t(kSharedStack) * threads * sizeof(uint2);
    // Fewer rays than the GPU holds at once: fewer of them in each warp.
    const uint32_t per_block = threads / 32, warps = uint32_t(c->sms) * 8u * per_block;
    if (const uint32_t quads = spread_quads(n, warps)) {
        const uint32_t grid = (n + per_block * quads - 1) / (per_block * quads);
        if (quant) k_closest_quad<true><<<grid, threads, smem, st>>>(c->scene(), V, rays, n, quads, hits);
        else k_closest_quad<false><<<grid, threads, smem, st>>>(c->scene(), V, rays, n, quads, hits);
        return cudaGetLastError();
    }
    const uint32_t lanes = spread_lanes(n, warps);
    const uint32_t grid = uint32_t((uint64_t(n) + per_block * lanes - 1) / (per_block * lanes));
    if (quant) {
        k_closest_fast<true><<<grid, threads, smem, st>>>(c->scene(), V, rays, n, lanes, hits);
    } else {
        k_closest_fast<false><<<grid, threads, smem, st>>>(c->scene(), V, rays, n, lanes, hits);
    }
    return cudaGetLastError();
}

}  // namespace ae

extern "C" int ae_build_wide_bvh(const ae_bvh_node *blas, uint32_t n_nodes, uint32_t tri_count, void *out_nodes,
                                 uint32_t capacity, uint32_t *out_count, uint32_t *out_root, int32_t *out_stack) {
    if (!blas || !out_count || !out_root || !out_stack) return AE_ERR_INVALID;
    std::vector<ae::WideNode> nodes;
    uint32_t root = 0;
    int stack = 0;
    std::string err;
    if (!ae::build_qbvh(blas, n_nodes, tri_count, nodes, root, stack, err)) {
        fprintf(stderr, "ae_build_wide_bvh: %s\n", err.c_str());
        return AE_ERR_LAYOUT;
    }
    *out_count = uint32_t(nodes.size());
    *out_root = root;
    *out_stack = stack;
    if (nodes.size() > capacity || (!out_nodes && !nodes.empty())) return AE_ERR_OVERSIZE;
    if (!nodes.empty()) std::memcpy(out_nodes, nodes.data(), nodes.size() * sizeof(ae::WideNode));
    return AE_OK;
}
