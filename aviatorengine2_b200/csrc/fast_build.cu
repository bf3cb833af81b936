// fast_build.cu - the optimised walks' mesh structures built on the device
// from the arrays that ae_upload_geometry already put there: the 4-wide nodes
// collapsed from the binary BLAS, the triangle records in leaf-slot order and
// the precision form's FP16 shading records.
//
// Collapse: a binary node becomes a 4-wide node when it is a tree's root or
// an interior child left after opening, of a node's two children, the
// interior one with the largest surface area until there are four (the rule
// of ae_build_wide_bvh).  Which nodes those are is found top down, one launch
// per tree level over all meshes together, with the level sizes kept on the
// device; a prefix sum over the marks numbers them in the binary order (depth
// first, so a subtree's nodes stay neighbours), and one pass writes them.
//
// On the host this took 0.35 us a triangle on one core (2.1M triangles: 0.7
// s of a context's preparation) before the copies of the results.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <tuple>
#include <utility>
#include <vector>

#include "context.h"
#include "fast.h"
#include "fast_trace.cuh"
#include "quantise.cuh"

namespace ae {

namespace {

constexpr int kMaxLevels = 32;  // uploads are checked to kBlasStack (24) pending nodes, so at most 23 levels
// Device words of a build: level sizes, then the flags below.
enum { W_STACK = kMaxLevels, W_ERROR, W_TOTAL, W_LOOSE, W_COUNT };
enum { E_LEAF = 1, E_QUANT = 2, E_SHARED = 4, E_DEPTH = 8 };

struct Kids {
    uint32_t k[4];
    int n;
};

// The intersection of a node's box and those above it.
struct Clip {
    float lo[3], hi[3];
};
__device__ Clip clip_to(const Clip &c, const ae_bvh_node &n) {
    const float lo[3] = {n.min_x, n.min_y, n.min_z}, hi[3] = {n.max_x, n.max_y, n.max_z};
    Clip r;
    for (int a = 0; a < 3; a++) {
        // A NaN bound stays, and holds nothing.
        r.lo[a] = lo[a] > c.lo[a] || lo[a] != lo[a] ? lo[a] : c.lo[a];
        r.hi[a] = hi[a] < c.hi[a] || hi[a] != hi[a] ? hi[a] : c.hi[a];
    }
    return r;
}

__device__ float node_half_area(const ae_bvh_node &n) {
    const float dx = __fsub_rn(n.max_x, n.min_x), dy = __fsub_rn(n.max_y, n.min_y), dz = __fsub_rn(n.max_z, n.min_z);
    return __fadd_rn(__fadd_rn(__fmul_rn(dx, dy), __fmul_rn(dy, dz)), __fmul_rn(dz, dx));
}

// The children of binary node i gathered into up to four.  clip (optional): on
// entry clip[0] is node i's, on return each child's.
__device__ Kids gather_kids(const ae_bvh_node *bin, uint32_t i, Clip *clip = nullptr) {
    Kids K;
    K.k[0] = uint32_t(bin[i].left);
    K.k[1] = uint32_t(bin[i].right);
    K.n = 2;
    if (clip) {
        clip[1] = clip_to(clip[0], bin[K.k[1]]);
        clip[0] = clip_to(clip[0], bin[K.k[0]]);
    }
    while (K.n < 4) {
        int best = -1;
        float area = -1.0f;
        for (int j = 0; j < K.n; j++) {
            if (bin[K.k[j]].count > 0) continue;
            const float a = node_half_area(bin[K.k[j]]);
            if (a > area) { area = a; best = j; }
        }
        if (best < 0) break;
        const uint32_t open = K.k[best];
        for (int j = K.n; j > best + 1; j--) {
            K.k[j] = K.k[j - 1];
            if (clip) clip[j] = clip[j - 1];
        }
        K.k[best] = uint32_t(bin[open].left);
        K.k[best + 1] = uint32_t(bin[open].right);
        if (clip) {
            clip[best + 1] = clip_to(clip[best], bin[K.k[best + 1]]);
            clip[best] = clip_to(clip[best], bin[K.k[best]]);
        }
        K.n++;
    }
    return K;
}

// A mesh: one grid row of the record kernels.
struct MeshJob {
    uint32_t vertex_base, index_base, tris, tri_base;
};
static_assert(sizeof(MeshJob) == 16, "four words in the build's tables");

// All trees of a build by first node, ascending, and the meshes of each: those
// numbered first_job[t] to first_job[t + 1].
struct Trees {
    const uint32_t *base, *first_job;
    uint32_t count;
    const MeshJob *jobs;
    const float4 *tris;
};

// Whether a leaf's triangles lie in the boxes above them, in every mesh that
// uses the tree (the exact walks count on it, exact_trace.cuh; the boxes of the
// nodes need not nest: flat ones are thicker than what they hold).
__device__ bool leaf_enclosed(const Trees &T, uint32_t base, const ae_bvh_node &leaf, const Clip &c) {
    uint32_t a = 0, b = T.count - 1;
    while (a < b) {
        const uint32_t m = (a + b) / 2;
        if (T.base[m] < base) a = m + 1;
        else b = m;
    }
    for (uint32_t j = T.first_job[a]; j < T.first_job[a + 1]; j++) {
        const MeshJob J = T.jobs[j];
        for (int32_t k = 0; k < leaf.count; k++) {
            if (uint32_t(leaf.left + k) >= J.tris) continue;
            const float4 *r = T.tris + 3 * (size_t(J.tri_base) + leaf.left + k);
            const float4 r0 = r[0], r1 = r[1], r2 = r[2];
            const float p[3][3] = {{r0.x, r0.y, r0.z}, {r0.w, r1.x, r1.y}, {r1.z, r1.w, r2.x}};
            for (int v = 0; v < 3; v++)
                for (int x = 0; x < 3; x++)
                    if (!(p[v][x] >= c.lo[x] && p[v][x] <= c.hi[x])) return false;
        }
    }
    return true;
}
__device__ Clip no_clip() {
    const float inf = __int_as_float(0x7f800000);
    return Clip{{-inf, -inf, -inf}, {inf, inf, inf}};
}

// Roots of the trees into the first level.  owner[i] is 1 + the tree's first
// node for the binary nodes that become 4-wide nodes, 0 for the rest.
__global__ void k_wide_roots(const ae_bvh_node *__restrict__ blas, const uint32_t *__restrict__ base, uint32_t trees,
                             uint32_t *owner, Clip *clips, uint2 *front, uint32_t *words) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= trees || blas[base[t]].count > 0) return;
    if (atomicExch(owner + base[t], base[t] + 1u)) {
        atomicOr(words + W_ERROR, uint32_t(E_SHARED));
        return;
    }
    clips[base[t]] = clip_to(no_clip(), blas[base[t]]);
    front[atomicAdd(words, 1u)] = make_uint2(base[t], 0u);
}

// One tree level: front entries are (binary node, stack entries that the walk
// holds when it reaches the node).
__global__ void __launch_bounds__(128) k_wide_level(const ae_bvh_node *__restrict__ blas, uint32_t *owner,
                                                    const uint2 *__restrict__ front, uint2 *__restrict__ next,
                                                    Clip *clips, Trees T, uint32_t *words, int level) {
    const uint32_t count = words[level];
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < count; j += gridDim.x * blockDim.x) {
        const uint32_t i = front[j].x, base = owner[i] - 1u;
        Clip clip[4];
        clip[0] = clips[i];
        const Kids K = gather_kids(blas + base, i - base, clip);
        const uint32_t need = front[j].y + uint32_t(K.n - 1);
        atomicMax(words + W_STACK, need);
        for (int k = 0; k < K.n; k++) {
            const uint32_t g = base + K.k[k];
            const ae_bvh_node &c = blas[g];
            if (c.count > 0) {
                if (uint32_t(c.count) > kMaxLeafCount || uint32_t(c.left) >= kMaxLeafFirst)
                    atomicOr(words + W_ERROR, uint32_t(E_LEAF));
                else if (!leaf_enclosed(T, base, c, clip[k])) words[W_LOOSE] = 1u;
                continue;
            }
            clips[g] = clip[k];
            if (atomicExch(owner + g, base + 1u)) atomicOr(words + W_ERROR, uint32_t(E_SHARED));
            else if (level + 1 <= kBlasStack) next[atomicAdd(words + level + 1, 1u)] = make_uint2(g, need);
            else atomicOr(words + W_ERROR, uint32_t(E_DEPTH));
        }
    }
}

// Exclusive prefix sum of (owner != 0): per block of 1024, then over the
// block sums.
__device__ uint32_t block_exclusive(uint32_t v, uint32_t *warp_sum, uint32_t &total) {
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    uint32_t incl = v;
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= uint32_t(off)) incl += y;
    }
    __syncthreads();
    if (lane == 31u) warp_sum[w] = incl;
    __syncthreads();
    uint32_t before = 0;
    total = 0;
    for (uint32_t j = 0; j < 32u; j++) {
        if (j < w) before += warp_sum[j];
        total += warp_sum[j];
    }
    return before + incl - v;
}
__global__ void __launch_bounds__(1024) k_wide_scan(const uint32_t *__restrict__ owner, uint32_t n,
                                                    uint32_t *__restrict__ index, uint32_t *__restrict__ sums) {
    __shared__ uint32_t ws[32];
    const uint32_t i = blockIdx.x * 1024u + threadIdx.x;
    uint32_t total;
    const uint32_t at = block_exclusive(i < n && owner[i] ? 1u : 0u, ws, total);
    if (i < n) index[i] = at;
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}
__global__ void __launch_bounds__(1024) k_wide_scan_sums(uint32_t *sums, uint32_t n, uint32_t *words) {
    __shared__ uint32_t ws[32];
    uint32_t before = 0;
    for (uint32_t b = 0; b < n; b += 1024u) {
        const uint32_t i = b + threadIdx.x;
        uint32_t total;
        const uint32_t at = block_exclusive(i < n ? sums[i] : 0u, ws, total);
        if (i < n) sums[i] = before + at;
        before += total;
    }
    if (threadIdx.x == 0) words[W_TOTAL] = before;
}

// Root references of the trees, first node offset by `first`.
__global__ void k_wide_root_refs(const ae_bvh_node *__restrict__ blas, const uint32_t *__restrict__ base,
                                 uint32_t trees, const uint32_t *__restrict__ index,
                                 const uint32_t *__restrict__ sums, uint32_t first, Trees T, uint32_t *words,
                                 uint32_t *__restrict__ ref) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= trees) return;
    const ae_bvh_node &r = blas[base[t]];
    if (r.count > 0) {
        if (uint32_t(r.count) > kMaxLeafCount || uint32_t(r.left) >= kMaxLeafFirst)
            atomicOr(words + W_ERROR, uint32_t(E_LEAF));
        else if (!leaf_enclosed(T, base[t], r, clip_to(no_clip(), r))) words[W_LOOSE] = 1u;
        ref[t] = leaf_ref(uint32_t(r.left) & 0xffffffu, uint32_t(r.count) & 0x7fu);
    } else {
        ref[t] = first + index[base[t]] + sums[base[t] >> 10];
    }
}

__global__ void __launch_bounds__(128) k_wide_emit(const ae_bvh_node *__restrict__ blas, uint32_t n,
                                                   const uint32_t *__restrict__ owner,
                                                   const uint32_t *__restrict__ index,
                                                   const uint32_t *__restrict__ sums, uint32_t first,
                                                   QNode *__restrict__ out, uint32_t *words) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !owner[i]) return;
    const uint32_t base = owner[i] - 1u;
    const Kids K = gather_kids(blas + base, i - base);
    QNode q;
    float box[4][6], u[6];
    bool valid[4];
    for (int k = 0; k < 4; k++) {
        valid[k] = k < K.n;
        q.child[k] = kNoChild;
        if (!valid[k]) continue;
        const uint32_t g = base + K.k[k];
        const ae_bvh_node c = blas[g];
        box[k][0] = c.min_x; box[k][1] = c.min_y; box[k][2] = c.min_z;
        box[k][3] = c.max_x; box[k][4] = c.max_y; box[k][5] = c.max_z;
        q.child[k] = c.count > 0 ? leaf_ref(uint32_t(c.left) & 0xffffffu, uint32_t(c.count) & 0x7fu)
                                 : first + index[g] + sums[g >> 10];
    }
    if (!quantise_node(q, K.n, box, valid, u)) atomicOr(words + W_ERROR, uint32_t(E_QUANT));
    out[first + index[i] + sums[i >> 10]] = q;
}

// Triangle records in slot order, one mesh per grid row.
__global__ void __launch_bounds__(256) k_tri_records(const ae_vertex *__restrict__ v, const uint32_t *__restrict__ idx,
                                                     const MeshJob *__restrict__ jobs, float4 *__restrict__ out,
                                                     uint32_t *most) {
    const MeshJob J = jobs[blockIdx.y];
    // Largest |e1| |e2| / |e1 x e2| of the triangles that the reference test can
    // accept (exact_trace.cuh), 1 and up; as bits, which order like the floats.
    uint32_t factor = 0;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < J.tris; t += gridDim.x * blockDim.x) {
        const uint32_t *ix = idx + J.index_base + 3u * t;
        const ae_vertex *a = v + J.vertex_base + ix[0], *b = v + J.vertex_base + ix[1], *c = v + J.vertex_base + ix[2];
        float4 *o = out + 3 * (size_t(J.tri_base) + t);
        o[0] = make_float4(a->px, a->py, a->pz, b->px);
        o[1] = make_float4(b->py, b->pz, c->px, c->py);
        o[2] = make_float4(c->pz, 0.0f, 0.0f, 0.0f);
        const f3 p0 = mk(a->px, a->py, a->pz), e1 = mk(b->px, b->py, b->pz) - p0, e2 = mk(c->px, c->py, c->pz) - p0;
        const f3 n = cross(e1, e2);
        const float nn = dot(n, n);
        if (!(nn < 1e-12f)) {
            const float f = sqrtf(dot(e1, e1)) * sqrtf(dot(e2, e2)) / sqrtf(nn);
            factor = max(factor, __float_as_uint(f >= 0.0f ? f : __int_as_float(0x7f800000)));
        }
    }
    factor = __reduce_max_sync(0xffffffffu, factor);
    if ((threadIdx.x & 31u) == 0 && factor) atomicMax(most, factor);
}

// FP16 shading records (layout in wf_common.cuh: PrecView).
__device__ uint32_t half2_bits(float lo, float hi) {
    return uint32_t(__half_as_ushort(__float2half_rn(lo))) | uint32_t(__half_as_ushort(__float2half_rn(hi))) << 16;
}
__global__ void __launch_bounds__(256) k_shade16(const ae_vertex *__restrict__ v, const uint32_t *__restrict__ idx,
                                                 const MeshJob *__restrict__ jobs, uint4 *__restrict__ out) {
    const MeshJob J = jobs[blockIdx.y];
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < J.tris; t += gridDim.x * blockDim.x) {
        const uint32_t *ix = idx + J.index_base + 3u * t;
        const ae_vertex a = v[J.vertex_base + ix[0]], b = v[J.vertex_base + ix[1]], c = v[J.vertex_base + ix[2]];
        uint4 *o = out + 2 * (size_t(J.tri_base) + t);
        o[0] = make_uint4(half2_bits(a.nx, a.ny), half2_bits(a.nz, b.nx), half2_bits(b.ny, b.nz), half2_bits(c.nx, c.ny));
        o[1] = make_uint4(half2_bits(c.nz, a.u), half2_bits(a.v, b.u), half2_bits(b.v, c.u), half2_bits(c.v, 0.0f));
    }
}

// Grid rows are meshes: launched in slices of at most 65,535.
template <class F> void for_rows(size_t rows, F launch) {
    for (size_t r = 0; r < rows; r += 65535) launch(r, uint32_t(std::min<size_t>(65535, rows - r)));
}

// The listed meshes by their trees' first nodes, and (optional) those.
std::vector<MeshJob> mesh_jobs(const FastScene &F, std::vector<uint32_t> *tree = nullptr) {
    std::vector<std::pair<uint32_t, MeshJob>> list;
    for (const auto &kv : F.mesh_roots)
        list.emplace_back(std::get<3>(kv.first), MeshJob{std::get<0>(kv.first), std::get<1>(kv.first), std::get<2>(kv.first),
                                                         kv.second.second});
    std::stable_sort(list.begin(), list.end(), [](const auto &a, const auto &b) { return a.first < b.first; });
    std::vector<MeshJob> jobs;
    for (const auto &x : list) {
        jobs.push_back(x.second);
        if (tree) tree->push_back(x.first);
    }
    return jobs;
}
uint32_t row_blocks(const std::vector<MeshJob> &jobs) {
    uint32_t most = 1;
    for (const MeshJob &j : jobs) most = std::max(most, j.tris);
    return std::min<uint32_t>((most + 255u) / 256u, 1u << 14);
}

}  // namespace

// Builds nodes and triangle records of every mesh listed in F.mesh_roots
// (their root references are filled in), replacing what was there.
int build_mesh_structures(Ctx *c, FastScene &F) {
    const uint32_t nb = uint32_t(c->n_blas);
    std::vector<uint32_t> bases, first_job, tree_of;
    const std::vector<MeshJob> jobs = mesh_jobs(F, &tree_of);
    for (size_t j = 0; j < jobs.size(); j++)
        if (!j || tree_of[j] != tree_of[j - 1]) {
            bases.push_back(tree_of[j]);
            first_job.push_back(uint32_t(j));
        }
    first_job.push_back(uint32_t(jobs.size()));
    F.max_stack = 0;
    F.n_nodes = 0;
    const uint32_t blocks = (nb + 1023u) / 1024u;
    if (F.tris.reserve(std::max<size_t>(size_t(F.n_tris) * 3, 1))) return c->fail(AE_ERR_OOM, "fast scene buffers");
    if (bases.empty()) return F.nodes.reserve(1) ? c->fail(AE_ERR_OOM, "fast scene buffers") : AE_OK;
    // One scratch allocation, freed on return: the host tables (jobs, roots, each
    // root's first job), then the build's arrays.
    const size_t at_base = jobs.size() * 4, at_first = at_base + bases.size(), at_refs = at_first + first_job.size(),
                 at_most = at_refs + bases.size(), at_words = at_most + 1, at_sums = at_words + W_COUNT,
                 at_owner = at_sums + blocks, at_index = at_owner + nb, at_clips = at_index + nb,
                 at_front = (at_clips + 6 * size_t(nb) + 1) & ~size_t(1);
    static_assert(sizeof(Clip) == 24, "six words a node");
    DevBuf<uint32_t> scratch;
    if (scratch.reserve(at_front + 4 * size_t(nb))) return c->fail(AE_ERR_OOM, "fast scene build scratch");
    const MeshJob *d_jobs = reinterpret_cast<const MeshJob *>(scratch.ptr);
    uint32_t *const d_base = scratch.ptr + at_base, *const refs = scratch.ptr + at_refs,
             *const words = scratch.ptr + at_words, *const sums = scratch.ptr + at_sums,
             *const owner = scratch.ptr + at_owner, *const index = scratch.ptr + at_index,
             *const most = scratch.ptr + at_most;
    Clip *const clips = reinterpret_cast<Clip *>(scratch.ptr + at_clips);
    const Trees T{d_base, scratch.ptr + at_first, uint32_t(bases.size()), d_jobs, F.tris.ptr};
    uint2 *const front = reinterpret_cast<uint2 *>(scratch.ptr + at_front);
    cudaStream_t st = c->stream;
    int rc;
    std::vector<uint32_t> tables(at_refs);
    std::memcpy(tables.data(), jobs.data(), jobs.size() * sizeof(MeshJob));
    std::copy(bases.begin(), bases.end(), tables.begin() + at_base);
    std::copy(first_job.begin(), first_job.end(), tables.begin() + at_first);
    if ((rc = c->cuda(cudaMemcpyAsync(scratch.ptr, tables.data(), at_refs * 4, cudaMemcpyHostToDevice, st), "mesh tables")) ||
        (rc = c->cuda(cudaMemsetAsync(most, 0, 4, st), "triangle factor")))
        return rc;
    const uint32_t gx = row_blocks(jobs);
    for_rows(jobs.size(), [&](size_t r, uint32_t rows) {
        k_tri_records<<<dim3(gx, rows), 256, 0, st>>>(c->vertices.ptr, c->indices.ptr, d_jobs + r, F.tris.ptr, most);
    });
    if ((rc = c->cuda(cudaGetLastError(), "triangle records"))) return rc;
    F.loose_trees = false;
    std::vector<uint32_t> host_refs(bases.size());
    // All trees in one build.  Trees that share nodes (one's root inside
    // another's range) are built one after another instead, each with its
    // own marks.
    size_t first_tree = 0, step = bases.size();
    while (first_tree < bases.size()) {
        const uint32_t trees = uint32_t(std::min(step, bases.size() - first_tree));
        const uint32_t *tb = d_base + first_tree;
        if ((rc = c->cuda(cudaMemsetAsync(owner, 0, size_t(nb) * 4, st), "marks")) ||
            (rc = c->cuda(cudaMemsetAsync(words, 0, W_COUNT * 4, st), "build words")))
            return rc;
        k_wide_roots<<<(trees + 127) / 128, 128, 0, st>>>(c->blas.ptr, tb, trees, owner, clips, front, words);
        for (int l = 0; l < kBlasStack + 1; l++)
            k_wide_level<<<c->sms * 4, 128, 0, st>>>(c->blas.ptr, owner, front + (l & 1 ? nb : 0),
                                                  front + (l & 1 ? 0 : nb), clips, T, words, l);
        k_wide_scan<<<blocks, 1024, 0, st>>>(owner, nb, index, sums);
        k_wide_scan_sums<<<1, 1024, 0, st>>>(sums, blocks, words);
        k_wide_root_refs<<<(trees + 127) / 128, 128, 0, st>>>(c->blas.ptr, tb, trees, index, sums, F.n_nodes,
                                                              T, words, refs + first_tree);
        uint32_t w[W_COUNT];
        if ((rc = c->cuda(cudaGetLastError(), "4-wide collapse")) ||
            (rc = c->cuda(cudaMemcpyAsync(w, words, sizeof(w), cudaMemcpyDeviceToHost, st), "build words")) ||
            (rc = c->cuda(cudaStreamSynchronize(st), "4-wide collapse")))
            return rc;
        if (w[W_ERROR] & E_LEAF) return c->fail(AE_ERR_LAYOUT, "4-wide BVH: leaf beyond the packed reference limits");
        if (w[W_ERROR] & E_DEPTH) return c->fail(AE_ERR_LAYOUT, "4-wide BVH: tree too deep");
        if (w[W_ERROR] & E_SHARED) {
            if (trees == 1) return c->fail(AE_ERR_LAYOUT, "4-wide BVH: node reached twice");
            F.n_nodes = 0;
            F.max_stack = 0;
            first_tree = 0;
            step = 1;
            continue;
        }
        if (w[W_STACK] + 1 > uint32_t(kFastStack))
            return c->fail(AE_ERR_LAYOUT, "4-wide BVH needs %u stack entries (> %d)", w[W_STACK] + 1, kFastStack);
        const size_t total = size_t(F.n_nodes) + w[W_TOTAL];
        if (F.nodes.cap < std::max<size_t>(total, 1)) {
            // Growing keeps the trees built before (one-by-one builds only).
            DevBuf<QNode> grown;
            if (grown.reserve(std::max<size_t>(step == 1 ? 2 * total : total, 1))) return c->fail(AE_ERR_OOM, "fast scene buffers");
            if (F.n_nodes && (rc = c->cuda(cudaMemcpyAsync(grown.ptr, F.nodes.ptr, size_t(F.n_nodes) * sizeof(QNode),
                                                           cudaMemcpyDeviceToDevice, st), "nodes")))
                return rc;
            if ((rc = c->cuda(cudaStreamSynchronize(st), "nodes"))) return rc;
            std::swap(F.nodes.ptr, grown.ptr);
            std::swap(F.nodes.cap, grown.cap);
        }
        k_wide_emit<<<(nb + 127) / 128, 128, 0, st>>>(c->blas.ptr, nb, owner, index, sums, F.n_nodes,
                                                      F.nodes.ptr, words);
        if ((rc = c->cuda(cudaGetLastError(), "4-wide nodes")) ||
            (rc = c->cuda(cudaMemcpyAsync(w, words, sizeof(w), cudaMemcpyDeviceToHost, st), "build words")) ||
            (rc = c->cuda(cudaStreamSynchronize(st), "4-wide nodes")))
            return rc;
        if (w[W_ERROR] & E_QUANT) return c->fail(AE_ERR_LAYOUT, "4-wide BVH: a child box cannot be quantised conservatively");
        F.loose_trees = F.loose_trees || w[W_LOOSE];
        F.n_nodes = uint32_t(total);
        F.max_stack = std::max(F.max_stack, int(w[W_STACK]));
        first_tree += trees;
    }
    uint32_t factor = 0;
    if ((rc = c->cuda(cudaMemcpyAsync(host_refs.data(), refs, bases.size() * 4, cudaMemcpyDeviceToHost, st), "tree roots")) ||
        (rc = c->cuda(cudaMemcpyAsync(&factor, most, 4, cudaMemcpyDeviceToHost, st), "triangle factor")) ||
        (rc = c->cuda(cudaStreamSynchronize(st), "triangle records")))
        return rc;
    std::memcpy(&F.tri_factor, &factor, 4);
    F.tri_factor = std::max(F.tri_factor, 1.0f);
    for (auto &kv : F.mesh_roots)
        kv.second.first = host_refs[std::lower_bound(bases.begin(), bases.end(), std::get<3>(kv.first)) - bases.begin()];
    return AE_OK;
}

// The precision form's shading records: per triangle, in the optimised
// BVH's slot order, the three vertex normals and UVs rounded to FP16
// (round to nearest even), 32 bytes.
int prepare_precision(Ctx *c) {
    int rc = prepare_fast(c);
    if (rc) return rc;
    FastScene &F = *c->fast;
    if (F.shade16_tris == F.n_tris && F.shade16.ptr) return AE_OK;
    const std::vector<MeshJob> jobs = mesh_jobs(F);
    DevBuf<MeshJob> d_jobs;
    if (F.shade16.reserve(size_t(std::max(F.n_tris, 1u)) * 2) || d_jobs.reserve(std::max<size_t>(jobs.size(), 1)))
        return c->fail(AE_ERR_OOM, "FP16 shading records");
    if (!jobs.empty() && (rc = c->cuda(cudaMemcpyAsync(d_jobs.ptr, jobs.data(), jobs.size() * sizeof(MeshJob),
                                                       cudaMemcpyHostToDevice, c->stream), "mesh jobs")))
        return rc;
    const uint32_t gx = row_blocks(jobs);
    for_rows(jobs.size(), [&](size_t r, uint32_t rows) {
        k_shade16<<<dim3(gx, rows), 256, 0, c->stream>>>(c->vertices.ptr, c->indices.ptr, d_jobs.ptr + r, F.shade16.ptr);
    });
    if ((rc = c->cuda(cudaGetLastError(), "FP16 shading records")) ||
        (rc = c->cuda(cudaStreamSynchronize(c->stream), "FP16 shading records")))
        return rc;
    F.shade16_tris = F.n_tris;
    return AE_OK;
}

}  // namespace ae
