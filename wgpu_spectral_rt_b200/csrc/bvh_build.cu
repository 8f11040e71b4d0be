// bvh_build.cu — GPU build of the compressed 8-wide BVH over the scene's
// flattened world-space triangles.
//
// Replaces the driver's BLAS/TLAS build (src/scene/builder.rs:131-266).
// Instances are flattened (their triangles transformed to world space) so a
// single tree serves every ray; shading still uses the instance's object
// space data.  Steps, all on the device:
//   1. flatten: world-space triangle slots + per-triangle instance id
//   2. centroid bounds and 30-bit Morton codes
//   3. radix sort of (code, triangle) pairs
//   4. binary radix tree over the sorted codes (Karras, HPG 2012)
//   5. bottom-up bounding boxes (one thread per leaf, atomic visit flags)
//   6. collapse into 8-wide nodes, level by level, of least surface-area cost
//      (collapse_costs); leaves hold at most leaf_max triangles (1..3, default
//      2); children are placed in slots by ray octant; child boxes are
//      quantised to 8 bits against the node's box.
#include <array>
#include <cmath>
#include <cstdio>
#include <string>
#include <vector>

#include "bvh_build.h"
#include "bvh_collapse.h"
#include "dev_arena.h"
#include "radix_sort.cuh"

namespace srt {

namespace {

constexpr uint32_t LEAF = 0x80000000u;
// A collapsed child with at most leaf_max triangles (BvhInputs) may become a
// leaf (its triangles listed in the node); larger ones become 8-wide nodes.
// At most 3: a node's leaves share a 24-bit triangle mask and a 5-bit offset
// field.  The closest hit is the minimum of (t, id) and an any-hit answer does
// not depend on the order, so the choice changes speed, never results.
constexpr uint32_t LEAF_MAX_LIMIT = 3u;

__device__ __forceinline__ uint32_t float_flip(float f) {
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float float_unflip(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

__global__ void k_flatten(const float4* __restrict__ vtx, const uint32_t* __restrict__ indices,
                          const uint4* __restrict__ mesh_infos, const InstDev* __restrict__ inst,
                          const InstFwd* __restrict__ fwd, uint32_t n_inst, uint32_t n_tris,
                          TriSlot* __restrict__ flat, uint32_t* __restrict__ tri_inst, float4* __restrict__ cen,
                          uint32_t* __restrict__ bounds /* 6 flipped: min xyz, max xyz */) {
    __shared__ uint32_t sb[6];
    if (threadIdx.x < 3) sb[threadIdx.x] = 0xFFFFFFFFu;
    else if (threadIdx.x < 6) sb[threadIdx.x] = 0u;
    __syncthreads();
    uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n_tris) {
        uint32_t lo = 0, hi = n_inst;  // last instance with tri_offset <= t
        while (hi - lo > 1) {
            uint32_t mid = (lo + hi) >> 1;
            if (inst[mid].tri_offset <= t) lo = mid;
            else hi = mid;
        }
        const InstDev& in = inst[lo];
        InstFwd f = fwd[lo];
        uint4 mi = mesh_infos[in.mesh_id];
        uint32_t io = mi.y + (t - in.tri_offset) * 3u;
        float3 w[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            float4 p = vtx[2 * (indices[io + k] + mi.x)];
            w[k] = xform_point(f, p.x, p.y, p.z);
        }
        TriSlot s;
        s.v0 = make_float4(w[0].x, w[0].y, w[0].z, __uint_as_float(t));
        s.v1 = make_float4(w[1].x, w[1].y, w[1].z, 0.f);
        s.v2 = make_float4(w[2].x, w[2].y, w[2].z, 0.f);
        flat[t] = s;
        tri_inst[t] = lo;
        float3 c = (w[0] + w[1] + w[2]) * (1.0f / 3.0f);
        cen[t] = make_float4(c.x, c.y, c.z, 0.f);
        atomicMin(&sb[0], float_flip(c.x));
        atomicMin(&sb[1], float_flip(c.y));
        atomicMin(&sb[2], float_flip(c.z));
        atomicMax(&sb[3], float_flip(c.x));
        atomicMax(&sb[4], float_flip(c.y));
        atomicMax(&sb[5], float_flip(c.z));
    }
    __syncthreads();
    if (threadIdx.x < 3) atomicMin(&bounds[threadIdx.x], sb[threadIdx.x]);
    else if (threadIdx.x < 6) atomicMax(&bounds[threadIdx.x], sb[threadIdx.x]);
}

__device__ __forceinline__ uint32_t expand_bits(uint32_t v) {
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}

__global__ void k_morton(const float4* __restrict__ cen, const uint32_t* __restrict__ bounds, uint32_t n,
                         uint32_t* __restrict__ keys, uint32_t* __restrict__ vals) {
    uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    float3 lo = f3(float_unflip(bounds[0]), float_unflip(bounds[1]), float_unflip(bounds[2]));
    float3 hi = f3(float_unflip(bounds[3]), float_unflip(bounds[4]), float_unflip(bounds[5]));
    float4 c = cen[t];
    float ex = fmaxf(hi.x - lo.x, 1e-30f), ey = fmaxf(hi.y - lo.y, 1e-30f), ez = fmaxf(hi.z - lo.z, 1e-30f);
    uint32_t x = (uint32_t)fminf(fmaxf((c.x - lo.x) / ex * 1024.0f, 0.0f), 1023.0f);
    uint32_t y = (uint32_t)fminf(fmaxf((c.y - lo.y) / ey * 1024.0f, 0.0f), 1023.0f);
    uint32_t z = (uint32_t)fminf(fmaxf((c.z - lo.z) / ez * 1024.0f, 0.0f), 1023.0f);
    keys[t] = (expand_bits(x) << 2) | (expand_bits(y) << 1) | expand_bits(z);
    vals[t] = t;
}

// delta(i, j): common prefix length of (key, index) pairs; -1 out of range.
__device__ __forceinline__ int delta(const uint32_t* keys, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    uint32_t a = keys[i], b = keys[j];
    if (a == b) return 32 + __clz((uint32_t)i ^ (uint32_t)j);
    return __clz(a ^ b);
}

struct Bvh2 {
    uint4* inode;      // internal: left ref, right ref, first, last
    float4* ibox;      // internal: lo, hi (2 per node)
    float4* lbox;      // leaf: lo, hi
    uint32_t* iparent; // parent of internal node
    uint32_t* lparent; // parent of leaf
    uint32_t* flags;   // refit visit counters
    float4* cost;      // internal: least costs of 1..7 wide roots below it (2 per node, see collapse_costs)
    uint2* choice;     // internal: what attains them, a byte each
};

// Which binary nodes become wide ones (bvh_collapse.h).
__device__ __forceinline__ void child_costs(const Bvh2& b, uint32_t ref, float4 lo, float4 hi, float* c) {
    if (ref & LEAF) {
        const float l = collapse_area(hi.x - lo.x, hi.y - lo.y, hi.z - lo.z) * COLLAPSE_TRI;
        for (int i = 0; i < 7; ++i) c[i] = l;
    } else {
        const float4 p = __ldcg(&b.cost[2 * ref]), q = __ldcg(&b.cost[2 * ref + 1]);
        c[0] = p.x;
        c[1] = p.y;
        c[2] = p.z;
        c[3] = p.w;
        c[4] = q.x;
        c[5] = q.y;
        c[6] = q.z;
    }
}
__device__ void collapse_costs(const Bvh2& b, uint32_t node, uint4 nd, float4 a0, float4 a1, float4 c0, float4 c1,
                               float4 lo, float4 hi, int width, uint32_t leaf_max) {
    float l[7], r[7], cost[7];
    uint32_t byte[8];
    child_costs(b, nd.x, a0, a1, l);
    child_costs(b, nd.y, c0, c1, r);
    collapse_choose(l, r, collapse_area(hi.x - lo.x, hi.y - lo.y, hi.z - lo.z), nd.w - nd.z + 1u, width, leaf_max, cost,
                    byte);
    b.cost[2 * node] = make_float4(cost[0], cost[1], cost[2], cost[3]);
    b.cost[2 * node + 1] = make_float4(cost[4], cost[5], cost[6], 0.f);
    b.choice[node] = make_uint2(byte[0] | (byte[1] << 8) | (byte[2] << 16) | (byte[3] << 24),
                                byte[4] | (byte[5] << 8) | (byte[6] << 16) | (byte[7] << 24));
}
__device__ __forceinline__ uint32_t choice_of(const Bvh2& b, uint32_t ref, int i) {  // i = 1 .. 8
    const uint2 c = b.choice[ref];
    return ((i <= 4 ? c.x >> (8 * (i - 1)) : c.y >> (8 * (i - 5)))) & 0xFFu;
}
struct Bvh2Tree {  // the binary tree as collapse_expand reads it
    const Bvh2& b;
    __device__ __forceinline__ bool leaf(uint32_t ref) const { return (ref & LEAF) != 0u; }
    __device__ __forceinline__ uint32_t left(uint32_t ref) const { return b.inode[ref].x; }
    __device__ __forceinline__ uint32_t right(uint32_t ref) const { return b.inode[ref].y; }
    __device__ __forceinline__ uint32_t choice(uint32_t ref, int i) const { return choice_of(b, ref, i); }
};

// Also looks at the sort that ordered the codes: where it gave up, keys and
// triangles may be anything, and nothing is built from them (ERR_WAIT_TIMEOUT).
__global__ void k_karras(const uint32_t* __restrict__ keys, int n, Bvh2 b, const uint32_t* __restrict__ sort_scratch,
                         uint32_t* __restrict__ err) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (sort_scratch[RS_GAVE_UP] != 0u) {
        if (i == 0) atomicOr(err, ERR_WAIT_TIMEOUT);
        return;
    }
    if (i >= n - 1) return;
    int d = (delta(keys, n, i, i + 1) - delta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
    int dmin = delta(keys, n, i, i - d);
    int lmax = 2;
    while (delta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
    int j = i + l * d;
    int dnode = delta(keys, n, i, j);
    int s = 0;
    int len = l;
    for (int t = (len + 1) >> 1;; t = (t + 1) >> 1) {
        if (delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
        if (t == 1) break;
    }
    int gamma = i + s * d + min(d, 0);
    int first = min(i, j), last = max(i, j);
    uint32_t left = (first == gamma) ? (LEAF | (uint32_t)gamma) : (uint32_t)gamma;
    uint32_t right = (last == gamma + 1) ? (LEAF | (uint32_t)(gamma + 1)) : (uint32_t)(gamma + 1);
    b.inode[i] = make_uint4(left, right, (uint32_t)first, (uint32_t)last);
    if (left & LEAF) b.lparent[left & ~LEAF] = (uint32_t)i;
    else b.iparent[left] = (uint32_t)i;
    if (right & LEAF) b.lparent[right & ~LEAF] = (uint32_t)i;
    else b.iparent[right] = (uint32_t)i;
}

__global__ void k_refit(const TriSlot* __restrict__ flat, const uint32_t* __restrict__ sorted_tri, int n, Bvh2 b,
                        int width, uint32_t leaf_max, const uint32_t* __restrict__ err) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || (*err & ERR_WAIT_TIMEOUT)) return;
    TriSlot s = flat[sorted_tri[i]];
    float3 lo = f3(fminf(fminf(s.v0.x, s.v1.x), s.v2.x), fminf(fminf(s.v0.y, s.v1.y), s.v2.y),
                   fminf(fminf(s.v0.z, s.v1.z), s.v2.z));
    float3 hi = f3(fmaxf(fmaxf(s.v0.x, s.v1.x), s.v2.x), fmaxf(fmaxf(s.v0.y, s.v1.y), s.v2.y),
                   fmaxf(fmaxf(s.v0.z, s.v1.z), s.v2.z));
    b.lbox[2 * i] = make_float4(lo.x, lo.y, lo.z, 0.f);
    b.lbox[2 * i + 1] = make_float4(hi.x, hi.y, hi.z, 0.f);
    if (n == 1) return;
    uint32_t node = b.lparent[i];
    while (true) {
        __threadfence();
        if (atomicAdd(&b.flags[node], 1u) == 0u) return;  // the sibling finishes this node
        __threadfence();
        uint4 nd = b.inode[node];
        float4 a0, a1, c0, c1;
        if (nd.x & LEAF) {
            a0 = __ldcg(&b.lbox[2 * (nd.x & ~LEAF)]);
            a1 = __ldcg(&b.lbox[2 * (nd.x & ~LEAF) + 1]);
        } else {
            a0 = __ldcg(&b.ibox[2 * nd.x]);
            a1 = __ldcg(&b.ibox[2 * nd.x + 1]);
        }
        if (nd.y & LEAF) {
            c0 = __ldcg(&b.lbox[2 * (nd.y & ~LEAF)]);
            c1 = __ldcg(&b.lbox[2 * (nd.y & ~LEAF) + 1]);
        } else {
            c0 = __ldcg(&b.ibox[2 * nd.y]);
            c1 = __ldcg(&b.ibox[2 * nd.y + 1]);
        }
        const float4 nlo = make_float4(fminf(a0.x, c0.x), fminf(a0.y, c0.y), fminf(a0.z, c0.z), 0.f);
        const float4 nhi = make_float4(fmaxf(a1.x, c1.x), fmaxf(a1.y, c1.y), fmaxf(a1.z, c1.z), 0.f);
        b.ibox[2 * node] = nlo;
        b.ibox[2 * node + 1] = nhi;
        collapse_costs(b, node, nd, a0, a1, c0, c1, nlo, nhi, width, leaf_max);
        if (node == 0u) return;
        node = b.iparent[node];
    }
}

// ---------------------------------------------------------------- binned SAH
// Top-down, one level of the binary tree per round: every node still to be
// split (a task: a contiguous range of the primitive permutation) bins its
// primitives' centroids into SAH_BINS bins along its widest centroid axis,
// picks the bin boundary of least surface-area cost N_L A_L + N_R A_R (a
// median split by position when all centroids share one bin, and for every
// node below SAH_MEDIAN_LEVEL levels, which bounds the depth), and
// partitions its range.  The result is the same binary tree format as the
// LBVH (internal nodes over contiguous ranges, single-primitive leaves), so
// the bottom-up box pass and the 8-wide collapse are shared.
// Bins per axis: SAH_BINS for ranges binned with atomics in global memory
// (more than SAH_SMALL primitives), SAH_LOCAL_BINS for the small ranges that
// their split warp bins in shared memory (2.5 KB per warp at 16, 10 KB at 64).
// Config 2 (1.57M triangles, leaves of <= 2): 16 / 16 bins 7.80 node visits
// per camera ray, closest hits 3.00 ms per 1080p frame; 64 / 16 7.18 visits,
// 2.86 ms; 64 / 32 and 64 / 64 within noise of 64 / 16 (2.85, 2.83 ms), and
// 128 / 16 of 64 / 16 (2.87 vs 2.88 ms); 96 / 16 7.45 visits, 2.91 ms.  The
// same hits in every case: the tree changes speed, never results.
#ifndef SRT_SAH_BINS
#define SRT_SAH_BINS 64
#endif
#ifndef SRT_SAH_LOCAL_BINS
#define SRT_SAH_LOCAL_BINS 16
#endif
constexpr int SAH_BINS = SRT_SAH_BINS;
constexpr int SAH_LOCAL_BINS = SRT_SAH_LOCAL_BINS;
static_assert(SAH_LOCAL_BINS <= SAH_BINS, "bin counts");
constexpr int SAH_REC = 13;  // count, box lo/hi, centroid lo/hi (flipped floats)
constexpr int SAH_TASK_WORDS = 3 * SAH_BINS * SAH_REC;  // bins of the three axes
constexpr int SAH_LOCAL_WORDS = 3 * SAH_LOCAL_BINS * SAH_REC;
constexpr uint32_t SAH_MEDIAN = 0xFFFFFFFFu;
constexpr uint32_t SAH_LOCAL = 0xFFFFFFFEu;  // binned by its split warp (small ranges)
constexpr uint32_t SAH_SMALL = 64;           // ranges up to this size bin without atomics
constexpr uint32_t SAH_MEDIAN_LEVEL = 48;

struct SahTask {
    uint32_t node, first, count, axis;
    float cmin[3], cscale[3];  // bin along axis a = (c_a - cmin[a]) * cscale[a]
    uint32_t nbins;            // bins per axis: SAH_BINS, or SAH_LOCAL_BINS for small ranges
    uint32_t bin_slot;         // bins of this task (SAH tasks only)
    uint32_t split, left_count;
    uint32_t lcur, rcur;
    uint32_t child_task[2];  // next-level task of each child, 0xFFFFFFFF for a leaf
};

__device__ __forceinline__ uint32_t sah_bin(const SahTask& t, float4 c, uint32_t ax) {
    float v = ax == 0 ? c.x : (ax == 1 ? c.y : c.z);
    float f = (v - t.cmin[ax]) * t.cscale[ax];
    int b = (int)f;
    return (uint32_t)min(max(b, 0), (int)t.nbins - 1);
}

__device__ __forceinline__ uint32_t sah_init_word(uint32_t i) {
    uint32_t k = i % SAH_REC;
    // lo fields start at +inf (min of flipped), hi fields at 0
    return (k == 0u) ? 0u : ((k >= 1 && k <= 3) || (k >= 7 && k <= 9)) ? 0xFFFFFFFFu : 0u;
}

__global__ void k_sah_init_bins(uint32_t* __restrict__ bins, uint32_t n_words) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_words) return;
    bins[i] = sah_init_word(i);
}

__device__ __forceinline__ void sah_accum(uint32_t* rec, float3 lo, float3 hi, float4 c) {
    atomicAdd(&rec[0], 1u);
    atomicMin(&rec[1], float_flip(lo.x));
    atomicMin(&rec[2], float_flip(lo.y));
    atomicMin(&rec[3], float_flip(lo.z));
    atomicMax(&rec[4], float_flip(hi.x));
    atomicMax(&rec[5], float_flip(hi.y));
    atomicMax(&rec[6], float_flip(hi.z));
    atomicMin(&rec[7], float_flip(c.x));
    atomicMin(&rec[8], float_flip(c.y));
    atomicMin(&rec[9], float_flip(c.z));
    atomicMax(&rec[10], float_flip(c.x));
    atomicMax(&rec[11], float_flip(c.y));
    atomicMax(&rec[12], float_flip(c.z));
}

// Bins of every active position (of tasks larger than SAH_SMALL) along all
// three axes; the tasks of the block's first and last positions (most of the
// block) aggregate in shared memory.
__global__ void k_sah_bin(const uint32_t* __restrict__ perm, const int* __restrict__ pos_task, uint32_t n,
                          const SahTask* __restrict__ tasks, const float4* __restrict__ cen,
                          const TriSlot* __restrict__ flat, uint32_t* __restrict__ bins) {
    __shared__ uint32_t sb[2][SAH_TASK_WORDS];
    __shared__ int ts[2];
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (threadIdx.x == 0) {
        ts[0] = pos_task[min(blockIdx.x * blockDim.x, n - 1)];
        ts[1] = pos_task[min(blockIdx.x * blockDim.x + blockDim.x - 1, n - 1)];
        if (ts[1] == ts[0]) ts[1] = -1;
        for (int k = 0; k < 2; ++k)
            if (ts[k] >= 0 && tasks[ts[k]].split != 0u) ts[k] = -1;
    }
    __syncthreads();
    for (int k = 0; k < 2; ++k)
        if (ts[k] >= 0)
            for (int i = threadIdx.x; i < SAH_TASK_WORDS; i += blockDim.x) sb[k][i] = sah_init_word((uint32_t)i);
    __syncthreads();
    if (p < n) {
        const int t = pos_task[p];
        if (t >= 0 && tasks[t].split == 0u) {
            const SahTask& T = tasks[t];
            const uint32_t prim = perm[p];
            const TriSlot s = flat[prim];
            const float3 lo = f3(fminf(fminf(s.v0.x, s.v1.x), s.v2.x), fminf(fminf(s.v0.y, s.v1.y), s.v2.y),
                                 fminf(fminf(s.v0.z, s.v1.z), s.v2.z));
            const float3 hi = f3(fmaxf(fmaxf(s.v0.x, s.v1.x), s.v2.x), fmaxf(fmaxf(s.v0.y, s.v1.y), s.v2.y),
                                 fmaxf(fmaxf(s.v0.z, s.v1.z), s.v2.z));
            const float4 c = cen[prim];
            uint32_t* dst = t == ts[0] ? sb[0] : t == ts[1] ? sb[1] : bins + (size_t)T.bin_slot * SAH_TASK_WORDS;
            for (uint32_t ax = 0; ax < 3; ++ax) {
                if (!(T.cscale[ax] > 0.f)) continue;
                sah_accum(dst + (ax * SAH_BINS + sah_bin(T, c, ax)) * SAH_REC, lo, hi, c);
            }
        }
    }
    __syncthreads();
    for (int k = 0; k < 2; ++k) {
        if (ts[k] < 0) continue;
        uint32_t* G = bins + (size_t)tasks[ts[k]].bin_slot * SAH_TASK_WORDS;
        for (int i = threadIdx.x; i < 3 * SAH_BINS; i += blockDim.x) {
            const uint32_t* r = sb[k] + i * SAH_REC;
            if (r[0] == 0u) continue;
            uint32_t* g = G + i * SAH_REC;
            atomicAdd(&g[0], r[0]);
            for (int j = 1; j <= 3; ++j) atomicMin(&g[j], r[j]);
            for (int j = 4; j <= 6; ++j) atomicMax(&g[j], r[j]);
            for (int j = 7; j <= 9; ++j) atomicMin(&g[j], r[j]);
            for (int j = 10; j <= 12; ++j) atomicMax(&g[j], r[j]);
        }
    }
}

__device__ __forceinline__ float half_area(float3 lo, float3 hi) {
    float3 e = f3(fmaxf(hi.x - lo.x, 0.f), fmaxf(hi.y - lo.y, 0.f), fmaxf(hi.z - lo.z, 0.f));
    return e.x * e.y + e.y * e.z + e.z * e.x;
}

// Sets the next-level task of one child: bin mappings of the three axes from
// its centroid bounds, and a bin slot when it will be binned.
__device__ void sah_child_task(SahTask& c, uint32_t node, uint32_t first, uint32_t count, float3 clo, float3 chi,
                               bool median, uint32_t* bin_alloc, uint32_t bin_cap) {
    c.node = node;
    c.first = first;
    c.count = count;
    const float lo[3] = {clo.x, clo.y, clo.z}, ext[3] = {chi.x - clo.x, chi.y - clo.y, chi.z - clo.z};
    bool any = false;
    for (int a = 0; a < 3; ++a) {
        c.cmin[a] = lo[a];
        c.cscale[a] = ext[a] > 0.f ? (float)(count <= SAH_SMALL ? SAH_LOCAL_BINS : SAH_BINS) / ext[a] : 0.f;
        any = any || ext[a] > 0.f;
    }
    c.axis = 0;
    c.nbins = count <= SAH_SMALL ? (uint32_t)SAH_LOCAL_BINS : (uint32_t)SAH_BINS;
    // all centroids on one point, below the SAH levels, or a range that the
    // collapse turns into one leaf anyway (<= 3): split by position
    c.split = (median || !any || count <= 3u) ? SAH_MEDIAN : (count <= SAH_SMALL ? SAH_LOCAL : 0u);
    c.bin_slot = 0xFFFFFFFFu;
    if (c.split == 0u) {
        uint32_t slot = atomicAdd(bin_alloc, 1u);
        if (slot < bin_cap) c.bin_slot = slot;
        else c.split = SAH_MEDIAN;  // out of bin slots (cannot happen: n / (SAH_SMALL + 1) tasks)
    }
    c.left_count = 0;
    c.lcur = c.rcur = 0;
    c.child_task[0] = c.child_task[1] = 0xFFFFFFFFu;
}

// One warp per task: choose the split (axis and bin boundary of least cost),
// create the children.  A lane holds SAH_PER consecutive bins of an axis: box
// and count of the bins before and after them come from shuffle scans, which
// give the same bits in any order (counts, minima and maxima), so the split is
// that of a serial sweep.  Small ranges bin here, in the warp's own shared
// memory.  With one thread per task (the sweep a chain of 13-word records in
// global memory, small ranges in a local array of 2.5 KB per thread) a level of
// a 630k-triangle scene took 0.315 ms instead of 0.041; a block's children take
// their nodes and tasks with one atomic each instead of one per child.
constexpr int SAH_SPLIT_WARPS = 8;
constexpr int SAH_PER = (SAH_BINS + 31) / 32;
struct SahRun {
    uint32_t n;
    float3 lo, hi;
};
__device__ __forceinline__ SahRun sah_none() {
    return SahRun{0u, f3(3.4e38f, 3.4e38f, 3.4e38f), f3(-3.4e38f, -3.4e38f, -3.4e38f)};
}
__device__ __forceinline__ SahRun sah_join(const SahRun& a, const SahRun& b) {
    return SahRun{a.n + b.n, f3(fminf(a.lo.x, b.lo.x), fminf(a.lo.y, b.lo.y), fminf(a.lo.z, b.lo.z)),
                  f3(fmaxf(a.hi.x, b.hi.x), fmaxf(a.hi.y, b.hi.y), fmaxf(a.hi.z, b.hi.z))};
}
// Exclusive scan over the warp's lanes, from lane 0 up or from lane 31 down.
template <bool UP>
__device__ __forceinline__ SahRun sah_scan(const SahRun& own, uint32_t lane) {
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    auto from = [](const SahRun& s, int d) {
        auto mv = [d](float v) { return UP ? __shfl_up_sync(FULL, v, d) : __shfl_down_sync(FULL, v, d); };
        return SahRun{UP ? __shfl_up_sync(FULL, s.n, d) : __shfl_down_sync(FULL, s.n, d),
                      f3(mv(s.lo.x), mv(s.lo.y), mv(s.lo.z)), f3(mv(s.hi.x), mv(s.hi.y), mv(s.hi.z))};
    };
    SahRun s = own;
#pragma unroll 1
    for (int d = 1; d < 32; d *= 2) {
        const SahRun o = from(s, d);
        if (UP ? lane >= (uint32_t)d : lane + d < 32u) s = sah_join(s, o);
    }
    const SahRun e = from(s, 1);
    return (UP ? lane == 0u : lane == 31u) ? sah_none() : e;
}

__global__ void __launch_bounds__(32 * SAH_SPLIT_WARPS)
    k_sah_split(SahTask* __restrict__ tasks, uint32_t n_tasks, const uint32_t* __restrict__ bins,
                const uint32_t* __restrict__ perm, const float4* __restrict__ cen, const TriSlot* __restrict__ flat,
                SahTask* __restrict__ next, uint32_t* __restrict__ n_next, uint32_t next_cap,
                uint32_t* __restrict__ bin_alloc, uint32_t bin_cap, uint32_t* __restrict__ node_alloc,
                uint32_t node_cap, Bvh2 b, uint32_t level, uint32_t* __restrict__ err) {
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    __shared__ uint32_t local[SAH_SPLIT_WARPS][SAH_LOCAL_WORDS];
    __shared__ uint32_t inner[SAH_SPLIT_WARPS];  // children of each warp's task that are nodes
    __shared__ uint32_t node_base, task_base;
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const uint32_t ti = blockIdx.x * SAH_SPLIT_WARPS + w;
    const bool valid = ti < n_tasks;
    SahTask& T = tasks[valid ? ti : 0u];  // (read and written by valid warps only)
    const uint32_t first = valid ? T.first : 0u, count = valid ? T.count : 2u, split = valid ? T.split : SAH_MEDIAN,
                   node = valid ? T.node : 0u;
    uint32_t left = count / 2;  // median by position
    float3 clo[2] = {f3(0.f, 0.f, 0.f), f3(0.f, 0.f, 0.f)}, chi[2] = {f3(0.f, 0.f, 0.f), f3(0.f, 0.f, 0.f)};
    bool median = split == SAH_MEDIAN;
    int bk = -1, bax = -1;
    if (!median) {
        const int NB = (int)T.nbins;  // the bin arrays' stride per axis
        const int per = (NB + 31) / 32;
        const uint32_t* Bt = local[w];
        if (split == 0u) {
            Bt = bins + (size_t)T.bin_slot * SAH_TASK_WORDS;
        } else {  // SAH_LOCAL
            for (uint32_t i = lane; i < (uint32_t)SAH_LOCAL_WORDS; i += 32u) local[w][i] = sah_init_word(i);
            __syncwarp();
            for (uint32_t q = first + lane; q < first + count; q += 32u) {
                const uint32_t prim = perm[q];
                const TriSlot s = flat[prim];
                const float4 c = cen[prim];
                const float3 lo = f3(fminf(fminf(s.v0.x, s.v1.x), s.v2.x), fminf(fminf(s.v0.y, s.v1.y), s.v2.y),
                                     fminf(fminf(s.v0.z, s.v1.z), s.v2.z));
                const float3 hi = f3(fmaxf(fmaxf(s.v0.x, s.v1.x), s.v2.x), fmaxf(fmaxf(s.v0.y, s.v1.y), s.v2.y),
                                     fmaxf(fmaxf(s.v0.z, s.v1.z), s.v2.z));
#pragma unroll 1
                for (uint32_t ax = 0; ax < 3; ++ax)
                    if (T.cscale[ax] > 0.f)
                        sah_accum(local[w] + (ax * SAH_LOCAL_BINS + sah_bin(T, c, ax)) * SAH_REC, lo, hi, c);
            }
            __syncwarp();
        }
        float best = 3.4e38f;
#pragma unroll 1
        for (int ax = 0; ax < 3; ++ax) {
            if (!(T.cscale[ax] > 0.f)) continue;
            const uint32_t* B = Bt + ax * NB * SAH_REC;
            SahRun bin[SAH_PER], own = sah_none();
#pragma unroll
            for (int j = 0; j < SAH_PER; ++j) {
                bin[j] = sah_none();
                const int k = (int)lane * per + j;
                if (j < per && k < NB) {
                    const uint32_t* r = B + k * SAH_REC;
                    if (r[0])
                        bin[j] = SahRun{r[0], f3(float_unflip(r[1]), float_unflip(r[2]), float_unflip(r[3])),
                                        f3(float_unflip(r[4]), float_unflip(r[5]), float_unflip(r[6]))};
                }
                own = sah_join(own, bin[j]);
            }
            SahRun l = sah_scan<true>(own, lane);
            const SahRun after = sah_scan<false>(own, lane);
            float cost = 3.4e38f;
            int ck = 0x7FFFFFFF;
#pragma unroll
            for (int j = 0; j < SAH_PER; ++j) {  // the boundary before the lane's bin j
                SahRun r = after;
#pragma unroll
                for (int i = SAH_PER - 1; i >= j; --i) r = sah_join(r, bin[i]);
                if (j < per && l.n && r.n) {
                    const float cj = (float)l.n * half_area(l.lo, l.hi) + (float)r.n * half_area(r.lo, r.hi);
                    if (cj < cost) {
                        cost = cj;
                        ck = (int)lane * per + j;
                    }
                }
                l = sah_join(l, bin[j]);
            }
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) {  // least cost, of equal ones the first boundary
                const float oc = __shfl_xor_sync(FULL, cost, d);
                const int ok = __shfl_xor_sync(FULL, ck, d);
                if (oc < cost || (oc == cost && ok < ck)) {
                    cost = oc;
                    ck = ok;
                }
            }
            if (cost < best) {
                best = cost;
                bk = ck;
                bax = ax;
            }
        }
        if (bk < 0) {
            median = true;
        } else {
            // the children's counts and centroid boxes (flipped floats order as integers)
            const uint32_t* B = Bt + bax * NB * SAH_REC;
            uint32_t n0 = 0u, lo[2][3], hi[2][3];
#pragma unroll
            for (int s = 0; s < 2; ++s)
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    lo[s][a] = 0xFFFFFFFFu;
                    hi[s][a] = 0u;
                }
            for (int k = (int)lane; k < NB; k += 32) {
                const uint32_t* r = B + k * SAH_REC;
                if (!r[0]) continue;
                const int side = k < bk ? 0 : 1;
                if (side == 0) n0 += r[0];
#pragma unroll
                for (int s = 0; s < 2; ++s)
#pragma unroll
                    for (int a = 0; a < 3; ++a)
                        if (side == s) {
                            lo[s][a] = min(lo[s][a], r[7 + a]);
                            hi[s][a] = max(hi[s][a], r[10 + a]);
                        }
            }
            left = __reduce_add_sync(FULL, n0);
#pragma unroll
            for (int s = 0; s < 2; ++s) {
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    lo[s][a] = __reduce_min_sync(FULL, lo[s][a]);
                    hi[s][a] = __reduce_max_sync(FULL, hi[s][a]);
                }
                clo[s] = f3(float_unflip(lo[s][0]), float_unflip(lo[s][1]), float_unflip(lo[s][2]));
                chi[s] = f3(float_unflip(hi[s][0]), float_unflip(hi[s][1]), float_unflip(hi[s][2]));
            }
        }
    }
    // centroid bounds are not tracked for position splits: the children keep
    // splitting by position
    const uint32_t n_inner = valid ? (left > 1u ? 1u : 0u) + (count - left > 1u ? 1u : 0u) : 0u;
    if (lane == 0u) inner[w] = n_inner;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t sum = 0u;
        for (int i = 0; i < SAH_SPLIT_WARPS; ++i) {
            const uint32_t n = inner[i];
            inner[i] = sum;
            sum += n;
        }
        node_base = sum ? atomicAdd(node_alloc, sum) : 0u;
        task_base = sum ? atomicAdd(n_next, sum) : 0u;
    }
    __syncthreads();
    if (!valid) return;
    uint32_t ref = 0u, child = 0xFFFFFFFFu;
    if (lane < 2u) {  // lane c makes child c
        const uint32_t cf = lane ? first + left : first, cc = lane ? count - left : left;
        if (cc == 1u) {
            ref = LEAF | cf;
            b.lparent[cf] = node;
        } else {
            const uint32_t rank = inner[w] + (lane && left > 1u ? 1u : 0u);
            const uint32_t nd = node_base + rank, tn = task_base + rank;
            if (nd >= node_cap || tn >= next_cap || cc == 0u) {
                atomicOr(err, ERR_QUEUE_OVERFLOW);
            } else {
                ref = nd;
                b.iparent[nd] = node;
                child = tn;
                sah_child_task(next[tn], nd, cf, cc, lane ? clo[1] : clo[0], lane ? chi[1] : chi[0],
                               median || level + 1 >= SAH_MEDIAN_LEVEL, bin_alloc, bin_cap);
            }
        }
        T.child_task[lane] = child;
    }
    const uint32_t ref1 = __shfl_sync(FULL, ref, 1);
    if (lane == 0u) {
        if (!median) T.axis = (uint32_t)bax;
        T.split = median ? SAH_MEDIAN : (uint32_t)bk;
        T.left_count = left;
        b.inode[node] = make_uint4(ref, ref1, first, first + count - 1u);
    }
}

__global__ void k_sah_root(const uint32_t* __restrict__ bounds, uint32_t n, SahTask* __restrict__ t,
                           int* __restrict__ pos_task, uint32_t* __restrict__ perm, uint32_t* __restrict__ bin_alloc,
                           uint32_t bin_cap) {
    uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p == 0) {
        float3 lo = f3(float_unflip(bounds[0]), float_unflip(bounds[1]), float_unflip(bounds[2]));
        float3 hi = f3(float_unflip(bounds[3]), float_unflip(bounds[4]), float_unflip(bounds[5]));
        sah_child_task(t[0], 0u, 0u, n, lo, hi, false, bin_alloc, bin_cap);
    }
    if (p < n) {
        pos_task[p] = 0;
        perm[p] = p;
    }
}

// Moves every active primitive into its child's range.  Lanes bound for the
// same child take their places with one atomic: a warp's positions are
// consecutive and mostly of one task, and 630k atomics on the two counters of
// the root took most of a level's time (0.082 -> 0.011 ms).
__global__ void k_sah_partition(const uint32_t* __restrict__ perm, const int* __restrict__ pos_task, uint32_t n,
                                SahTask* __restrict__ tasks, const float4* __restrict__ cen,
                                uint32_t* __restrict__ perm2, int* __restrict__ pos_task2) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    const int t = p < n ? pos_task[p] : -1;
    const uint32_t prim = p < n ? perm[p] : 0u;
    const uint32_t active = __ballot_sync(0xFFFFFFFFu, t >= 0);
    if (p >= n) return;
    if (t < 0) {
        perm2[p] = prim;
        pos_task2[p] = -1;
        return;
    }
    SahTask& T = tasks[t];
    uint32_t side;
    if (T.split == SAH_MEDIAN) side = (p - T.first) >= T.left_count ? 1u : 0u;
    else side = sah_bin(T, cen[prim], T.axis) >= T.split ? 1u : 0u;
    const uint32_t same = __match_any_sync(active, 2u * (uint32_t)t + side);
    const uint32_t lane = threadIdx.x & 31u;
    const int leader = __ffs(same) - 1;
    uint32_t base = 0u;
    if ((int)lane == leader) base = atomicAdd(side ? &T.rcur : &T.lcur, (uint32_t)__popc(same));
    base = __shfl_sync(same, base, leader) + __popc(same & ((1u << lane) - 1u));
    const uint32_t np = T.first + (side ? T.left_count : 0u) + base;
    perm2[np] = prim;
    pos_task2[np] = T.child_task[side] == 0xFFFFFFFFu ? -1 : (int)T.child_task[side];
}

__device__ __forceinline__ void ref_box(const Bvh2& b, uint32_t r, float3& lo, float3& hi) {
    float4 a, c;
    if (r & LEAF) {
        a = b.lbox[2 * (r & ~LEAF)];
        c = b.lbox[2 * (r & ~LEAF) + 1];
    } else {
        a = b.ibox[2 * r];
        c = b.ibox[2 * r + 1];
    }
    lo = xyz(a);
    hi = xyz(c);
}
__device__ __forceinline__ void ref_range(const Bvh2& b, uint32_t r, uint32_t& first, uint32_t& count) {
    if (r & LEAF) {
        first = r & ~LEAF;
        count = 1;
    } else {
        uint4 nd = b.inode[r];
        first = nd.z;
        count = nd.w - nd.z + 1;
    }
}

// Quantisation frame and 8-bit child boxes of one node, children indexed by
// slot (slots outside `used` empty): writes nd.a (origin, exponent bytes,
// imask), nd.c, nd.d, nd.e.  250 quanta span the node; the origin sits two
// quanta below it, and every child plane is padded outward by one quantum,
// which covers the half-quantum error of the traversal's biased-byte
// evaluation (see traverse<> in device_common.cuh).
__device__ void quantize_node(float3 nlo, float3 nhi, const float3* slo, const float3* shi, uint32_t used,
                              uint32_t imask, Node8& nd, uint32_t* err) {
    uint32_t ebyte[3];
    float scale[3];
    float nlov[3] = {nlo.x, nlo.y, nlo.z}, nhiv[3] = {nhi.x, nhi.y, nhi.z};
    for (int a = 0; a < 3; ++a) {
        double ext = (double)nhiv[a] - (double)nlov[a];
        int ex = -126;
        if (ext > 0.0) {
            ex = (int)ceil(log2(ext / 250.0));
            if (ldexp(250.0, ex) < ext) ++ex;
        }
        // a quantum of at least 4 float ulps of the node's coordinates, so the
        // shifted origin below stays exact to a quarter quantum
        double mag = fmax(fabs((double)nlov[a]), fabs((double)nhiv[a]));
        ex = max(ex, (int)ceil(log2(fmax(mag, 1e-30) * 4.0 / 8388608.0)));
        ex = max(ex, -126);
        ex = min(ex, 127);
        ebyte[a] = (uint32_t)(ex + 127);
        scale[a] = __uint_as_float(ebyte[a] << 23);
        double lo_exact = (double)nlov[a];
        nlov[a] = (float)(lo_exact - 2.0 * (double)scale[a]);
        // (to -infinity: towards a finite end a corner near -3.4e38 would move away from it for good)
        while ((double)nlov[a] > lo_exact - 2.0 * (double)scale[a])
            nlov[a] = nextafterf(nlov[a], __int_as_float(0xFF800000));
    }
    uint32_t qlo[3][2] = {{0u, 0u}, {0u, 0u}, {0u, 0u}}, qhi[3][2] = {{0u, 0u}, {0u, 0u}, {0u, 0u}};
    for (int s = 0; s < 8; ++s) {
        if (!((used >> s) & 1u)) continue;
        float lo3[3] = {slo[s].x, slo[s].y, slo[s].z}, hi3[3] = {shi[s].x, shi[s].y, shi[s].z};
        for (int a = 0; a < 3; ++a) {
            double sc = (double)scale[a];
            // one quantum of padding on each side
            int ql = (int)fmin(fmax(floor(((double)lo3[a] - (double)nlov[a]) / sc) - 1.0, 0.0), 255.0);
            int qh = (int)fmin(fmax(ceil(((double)hi3[a] - (double)nlov[a]) / sc) + 1.0, 0.0), 255.0);
            while (ql > 0 && (double)nlov[a] + ql * sc > (double)lo3[a] - sc) --ql;
            while (qh < 255 && (double)nlov[a] + qh * sc < (double)hi3[a] + sc) ++qh;
            if ((double)nlov[a] + ql * sc > (double)lo3[a] - sc || (double)nlov[a] + qh * sc < (double)hi3[a] + sc)
                atomicOr(err, ERR_BAD_INDEX);  // the frame cannot hold the padded child: reject the tree
            qlo[a][s >> 2] |= (uint32_t)ql << (8 * (s & 3));
            qhi[a][s >> 2] |= (uint32_t)qh << (8 * (s & 3));
        }
    }
    nd.a = make_uint4(__float_as_uint(nlov[0]), __float_as_uint(nlov[1]), __float_as_uint(nlov[2]),
                      ebyte[0] | (ebyte[1] << 8) | (ebyte[2] << 16) | (imask << 24));
    nd.c = make_uint4(qlo[0][0], qlo[0][1], qlo[1][0], qlo[1][1]);
    nd.d = make_uint4(qlo[2][0], qlo[2][1], qhi[0][0], qhi[0][1]);
    nd.e = make_uint4(qhi[1][0], qhi[1][1], qhi[2][0], qhi[2][1]);
}

// Refit of one level's nodes: child boxes from the deeper level's results
// (aux) or from the leaf triangles, then the node's frame is re-quantised.
__global__ void k_refit8(Node8* __restrict__ nodes, const TriSlot* __restrict__ tris, uint32_t begin, uint32_t end,
                         float4* __restrict__ aux, uint32_t* __restrict__ err) {
    uint32_t i = begin + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= end) return;
    Node8 nd = nodes[i];
    const uint32_t imask = nd.a.w >> 24, child_base = nd.b.x, tri_base = nd.b.y;
    const uint32_t meta[2] = {nd.b.z, nd.b.w};
    float3 slo[8], shi[8];
    float3 nlo = f3(3.4e38f, 3.4e38f, 3.4e38f), nhi = f3(-3.4e38f, -3.4e38f, -3.4e38f);
    uint32_t used = 0u;
    for (int s = 0; s < 8; ++s) {
        const uint32_t m = (meta[s >> 2] >> (8 * (s & 3))) & 0xFFu;
        if (m == 0u) continue;
        used |= 1u << s;
        float3 lo, hi;
        if ((imask >> s) & 1u) {
            const uint32_t child = child_base + __popc(imask & ((1u << s) - 1u));
            float4 a = aux[2 * child], b = aux[2 * child + 1];
            lo = f3(a.x, a.y, a.z);
            hi = f3(b.x, b.y, b.z);
        } else {
            lo = f3(3.4e38f, 3.4e38f, 3.4e38f);
            hi = f3(-3.4e38f, -3.4e38f, -3.4e38f);
            const uint32_t cnt = m >> 5, off = m & 31u;
            for (uint32_t k = 0; k < cnt; ++k) {
                const TriSlot& t = tris[tri_base + off + k];
                float3 v[3] = {f3(t.v0.x, t.v0.y, t.v0.z), f3(t.v1.x, t.v1.y, t.v1.z), f3(t.v2.x, t.v2.y, t.v2.z)};
                for (int j = 0; j < 3; ++j) {
                    lo = f3(fminf(lo.x, v[j].x), fminf(lo.y, v[j].y), fminf(lo.z, v[j].z));
                    hi = f3(fmaxf(hi.x, v[j].x), fmaxf(hi.y, v[j].y), fmaxf(hi.z, v[j].z));
                }
            }
        }
        slo[s] = lo;
        shi[s] = hi;
        nlo = f3(fminf(nlo.x, lo.x), fminf(nlo.y, lo.y), fminf(nlo.z, lo.z));
        nhi = f3(fmaxf(nhi.x, hi.x), fmaxf(nhi.y, hi.y), fmaxf(nhi.z, hi.z));
    }
    aux[2 * i] = make_float4(nlo.x, nlo.y, nlo.z, 0.f);
    aux[2 * i + 1] = make_float4(nhi.x, nhi.y, nhi.z, 0.f);
    quantize_node(nlo, nhi, slo, shi, used, imask, nd, err);
    nodes[i] = nd;
}

// Scatter masks of one level's nodes, from the deeper level's masks or the leaf triangles' materials.
__global__ void k_scatter_mask(const Node8* __restrict__ nodes, const TriSlot* __restrict__ tris,
                               const uint32_t* __restrict__ tri_inst, const InstDev* __restrict__ inst,
                               const float4* __restrict__ materials, uint32_t begin, uint32_t end,
                               uint8_t* __restrict__ mask) {
    const uint32_t i = begin + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= end) return;
    const uint32_t imask = nodes[i].a.w >> 24;
    const uint4 b = nodes[i].b;
    uint32_t out = 0u;
    for (uint32_t s = 0; s < 8u; ++s) {
        const uint32_t m = ((s < 4u ? b.z : b.w) >> (8u * (s & 3u))) & 0xFFu;
        if (m == 0u) continue;
        bool any = false;
        if ((imask >> s) & 1u) {
            any = mask[b.x + __popc(imask & ((1u << s) - 1u))] != 0u;
        } else {
            for (uint32_t k = 0; k < (m >> 5); ++k) {
                const uint32_t tri = __float_as_uint(tris[b.y + (m & 31u) + k].v0.w);
                any = any || scatters_photons(materials[2 * inst[tri_inst[tri]].mat_id + 1]);
            }
        }
        if (any) out |= 1u << s;
    }
    mask[i] = (uint8_t)out;
}

// Leaf slots of moved instances, re-transformed from object space.
__global__ void k_update_slots(TriSlot* __restrict__ tris, uint32_t n_tris, const uint32_t* __restrict__ tri_inst,
                               const uint8_t* __restrict__ moved, const float4* __restrict__ vtx,
                               const uint32_t* __restrict__ indices, const uint4* __restrict__ mesh_infos,
                               const InstDev* __restrict__ inst, const InstFwd* __restrict__ fwd) {
    uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n_tris) return;
    TriSlot s = tris[k];
    const uint32_t t = __float_as_uint(s.v0.w);
    const uint32_t ii = tri_inst[t];
    if (!moved[ii]) return;
    const InstDev& in = inst[ii];
    const InstFwd f = fwd[ii];
    const uint4 mi = mesh_infos[in.mesh_id];
    const uint32_t io = mi.y + (t - in.tri_offset) * 3u;
    float3 w[3];
    for (int j = 0; j < 3; ++j) {
        float4 p = vtx[2 * (indices[io + j] + mi.x)];
        w[j] = xform_point(f, p.x, p.y, p.z);
    }
    s.v0 = make_float4(w[0].x, w[0].y, w[0].z, s.v0.w);
    s.v1 = make_float4(w[1].x, w[1].y, w[1].z, 0.f);
    s.v2 = make_float4(w[2].x, w[2].y, w[2].z, 0.f);
    tris[k] = s;
}

// One block per light instance: its triangles in world space
// (builder.rs:101-129; w = 1, params copied).
__global__ void k_expand_lights(const LightInst* __restrict__ li, const uint8_t* __restrict__ moved,
                                const float4* __restrict__ vtx, const uint32_t* __restrict__ indices,
                                const uint4* __restrict__ mesh_infos, const InstDev* __restrict__ inst,
                                const InstFwd* __restrict__ fwd, float4* __restrict__ lights) {
    const LightInst L = li[blockIdx.x];
    if (moved && !moved[L.inst]) return;
    const InstDev& in = inst[L.inst];
    const InstFwd f = fwd[L.inst];
    const uint4 mi = mesh_infos[in.mesh_id];
    for (uint32_t k = threadIdx.x; k < L.count; k += blockDim.x) {
        float4* o = lights + 4ull * (L.first + k);
        for (int j = 0; j < 3; ++j) {
            float4 p = vtx[2 * (indices[mi.y + 3u * k + j] + mi.x)];
            float3 w = xform_point(f, p.x, p.y, p.z);
            o[j] = make_float4(w.x, w.y, w.z, 1.0f);
        }
        o[3] = L.params;
    }
}

// One thread per 8-wide node of this level: queue entries (bvh2 ref, node).
// Nodes over more than `open_above` triangles open their largest children.
__global__ void k_collapse(Bvh2 b, const uint2* __restrict__ qin, uint32_t n_in, uint2* __restrict__ qout,
                           uint32_t* __restrict__ n_out, Node8* __restrict__ nodes, uint32_t* __restrict__ node_alloc,
                           uint32_t node_cap, TriSlot* __restrict__ tris_out, uint32_t* __restrict__ tri_alloc,
                           uint32_t tri_cap, const TriSlot* __restrict__ flat, const uint32_t* __restrict__ sorted_tri,
                           uint32_t* __restrict__ err, int width, uint32_t leaf_max, uint32_t open_above) {
    uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n_in || (*(volatile uint32_t*)err & ERR_WAIT_TIMEOUT)) return;
    uint2 q = qin[e];
    uint32_t refs[8];
    int nc = 1;
    refs[0] = q.x;
    const uint32_t below = (q.x & LEAF) ? 1u : b.inode[q.x].w - b.inode[q.x].z + 1u;
    if (!(q.x & LEAF) && below > open_above) {
        // the child of largest area opened until the node is full: a node over
        // more than half of the triangles, or every one (build_bvh8).  The recurrence would make the big flat
        // leaves (walls) its children, where the quanta are coarsest and every
        // ray that starts on a wall meets its box: with it at the root too,
        // bounce 0 of config 2 0.342 vs 0.325 ms, its shadow rays 1.94 vs 1.87 ms
        // per frame, prism 96x64 camera rays 38 vs 33 us and shadow rays 20 vs
        // 12 us (opened down to n / 8 or n / 64 triangles: config 2 shadow rays
        // 1.88, 1.89 ms, closest hits 3.26, 3.27 vs 3.22).
        uint4 nd = b.inode[q.x];
        refs[0] = nd.x;
        refs[1] = nd.y;
        nc = 2;
        while (nc < width) {
            int best = -1;
            float best_area = -1.0f;
            for (int c = 0; c < nc; ++c) {
                if (refs[c] & LEAF) continue;
                float3 lo, hi;
                ref_box(b, refs[c], lo, hi);
                const float area = half_area(lo, hi);
                if (area > best_area) {
                    best_area = area;
                    best = c;
                }
            }
            if (best < 0) break;
            nd = b.inode[refs[best]];
            refs[best] = nd.x;
            refs[nc++] = nd.y;
        }
    } else if (!(q.x & LEAF)) {
        bool ok = true;
        nc = collapse_expand(Bvh2Tree{b}, q.x, width, refs, ok);
        if (!ok) atomicOr(err, ERR_BAD_INDEX);
    }
    // children boxes, counts and node box
    float3 clo[8], chi[8];
    uint32_t cfirst[8], ccount[8];
    float3 nlo = f3(3.4e38f, 3.4e38f, 3.4e38f), nhi = f3(-3.4e38f, -3.4e38f, -3.4e38f);
    uint32_t n_int = 0, n_tri = 0;
    bool is_leaf[8];
    for (int c = 0; c < nc; ++c) {
        ref_box(b, refs[c], clo[c], chi[c]);
        ref_range(b, refs[c], cfirst[c], ccount[c]);
        nlo = f3(fminf(nlo.x, clo[c].x), fminf(nlo.y, clo[c].y), fminf(nlo.z, clo[c].z));
        nhi = f3(fmaxf(nhi.x, chi[c].x), fmaxf(nhi.y, chi[c].y), fmaxf(nhi.z, chi[c].z));
        is_leaf[c] = (refs[c] & LEAF) ||
                     (ccount[c] <= leaf_max && (open_above == 0u || choice_of(b, refs[c], 1) != 0u));
        if (is_leaf[c]) n_tri += ccount[c];
        else ++n_int;
    }
    uint32_t child_base = n_int ? atomicAdd(node_alloc, n_int) : 0u;
    uint32_t tri_base = n_tri ? atomicAdd(tri_alloc, n_tri) : 0u;
    if (child_base + n_int > node_cap || tri_base + n_tri > tri_cap) {
        atomicOr(err, ERR_QUEUE_OVERFLOW);
        return;
    }
    const float3 pc = (nlo + nhi) * 0.5f;
    float from_centre[8][3];
    int child_in[8];
    for (int c = 0; c < nc; ++c) {
        const float3 d = (clo[c] + chi[c]) * 0.5f - pc;
        from_centre[c][0] = d.x;
        from_centre[c][1] = d.y;
        from_centre[c][2] = d.z;
    }
    collapse_slots(nc, from_centre, child_in);
    uint32_t meta[2] = {0u, 0u};
    uint32_t imask = 0u, int_rank = 0u, tri_off = 0u, used = 0u;
    float3 slo[8], shi[8];
    for (int s = 0; s < 8; ++s) {
        int c = child_in[s];
        if (c < 0) continue;
        used |= 1u << s;
        slo[s] = clo[c];
        shi[s] = chi[c];
        uint32_t m;
        if (is_leaf[c]) {
            m = (ccount[c] << 5) | tri_off;
            for (uint32_t k = 0; k < ccount[c]; ++k) tris_out[tri_base + tri_off + k] = flat[sorted_tri[cfirst[c] + k]];
            tri_off += ccount[c];
        } else {
            m = 7u << 5;
            imask |= 1u << s;
            uint32_t slot = atomicAdd(n_out, 1u);
            qout[slot] = make_uint2(refs[c], child_base + int_rank);
            ++int_rank;
        }
        meta[s >> 2] |= m << (8 * (s & 3));
    }
    Node8 nd;
    quantize_node(nlo, nhi, slo, shi, used, imask, nd, err);
    nd.b = make_uint4(child_base, tri_base, meta[0], meta[1]);
    nodes[q.y] = nd;
}

}  // namespace

cudaError_t build_bvh8(const BvhInputs& in, cudaStream_t st, BvhOutputs* out, std::string* msg) {
    uint32_t n = in.n_tris;
    out->nodes = nullptr;
    out->tris = nullptr;
    out->tri_inst = nullptr;
    out->scatter = nullptr;
    out->mem = nullptr;
    out->n_nodes = 0;
    out->depth = 0;
    out->kernel_launches = 0;
    cudaError_t e = cudaSuccess;
#define CK(x)                                         \
    do {                                              \
        e = (x);                                      \
        if (e != cudaSuccess) {                       \
            if (msg) *msg = std::string(#x) + ": " + cudaGetErrorString(e); \
            goto done;                                \
        }                                             \
    } while (0)
    TriSlot* flat = nullptr;
    float4* cen = nullptr;
    uint32_t *bounds = nullptr, *keys = nullptr, *vals = nullptr, *keys2 = nullptr, *vals2 = nullptr,
             *scratch = nullptr, *counters = nullptr, *err = nullptr;
    uint2 *qa = nullptr, *qb = nullptr;
    SahTask* sah_tasks[2] = {nullptr, nullptr};
    uint32_t* sah_bins = nullptr;
    Bvh2 b{};
    // two allocations instead of 30: 13 of the 32 ms that the build of a
    // 630k-triangle tree took were cudaMalloc and cudaFree
    DevArena kept, tmp;
    if (n == 0) return cudaSuccess;
    {
        const uint32_t node_cap = n > 1 ? n - 1 : 1;
        kept.add(&out->tri_inst, n);
        kept.add(&out->tris, n);
        kept.add(&out->nodes, node_cap);
        kept.add(&out->scatter, node_cap);
        CK(kept.commit());
        tmp.add(&flat, n);
        tmp.add(&cen, n);
        tmp.add(&bounds, 6);
        tmp.add(&keys, n);
        tmp.add(&vals, n);
        tmp.add(&keys2, n);
        tmp.add(&vals2, n);
        tmp.add(&scratch, radix_scratch_words(n));
        tmp.add(&counters, 4);
        tmp.add(&err, 1);
        tmp.add(&qa, node_cap);
        tmp.add(&qb, node_cap);
        tmp.add(&b.inode, node_cap);
        tmp.add(&b.ibox, 2 * (size_t)node_cap);
        tmp.add(&b.lbox, 2 * (size_t)n);
        tmp.add(&b.iparent, node_cap);
        tmp.add(&b.lparent, n);
        tmp.add(&b.flags, node_cap);
        tmp.add(&b.cost, 2 * (size_t)node_cap);
        tmp.add(&b.choice, node_cap);
        const bool sah = in.builder != BVH_BUILDER_LBVH && n >= 2;
        const uint32_t task_cap = n / 2 + 1;
        // tasks that bin in global memory hold more than SAH_SMALL primitives
        // of disjoint ranges: at most n / (SAH_SMALL + 1) per level
        const uint32_t bin_cap = n / (SAH_SMALL + 1) + 1;
        if (sah) {
            tmp.add(&sah_tasks[0], task_cap);
            tmp.add(&sah_tasks[1], task_cap);
            tmp.add(&sah_bins, (size_t)bin_cap * SAH_TASK_WORDS);
        }
        CK(tmp.commit());
        uint32_t init_bounds[6] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u, 0u};
        CK(cudaMemcpyAsync(bounds, init_bounds, sizeof(init_bounds), cudaMemcpyHostToDevice, st));
        CK(cudaMemsetAsync(b.flags, 0, sizeof(uint32_t) * node_cap, st));
        CK(cudaMemsetAsync(err, 0, 4, st));
        const int B = 256;
        uint32_t grid = (n + B - 1) / B;
        k_flatten<<<grid, B, 0, st>>>(in.vtx, in.indices, in.mesh_infos, in.inst, in.fwd, in.n_inst, n, flat,
                                      out->tri_inst, cen, bounds);
        ++out->kernel_launches;
        uint32_t* sv = nullptr;
        if (!sah) {
            k_morton<<<grid, B, 0, st>>>(cen, bounds, n, keys, vals);
            ++out->kernel_launches;
            uint32_t* sk;
            out->kernel_launches += sort_pairs(keys, vals, keys2, vals2, n, nullptr, 0, 30, scratch, st, &sk, &sv);
            if (n > 1) {
                k_karras<<<(n - 1 + B - 1) / B, B, 0, st>>>(sk, (int)n, b, scratch, err);
                ++out->kernel_launches;
            }
        } else {
            // binned SAH, level by level (keys/vals/keys2/vals2 serve as the
            // permutation and position -> task ping-pong buffers)
            uint32_t *perm = keys, *perm2 = keys2;
            int *pt = (int*)vals, *pt2 = (int*)vals2;
            // counters: node alloc, -, next tasks, bin slots of the next level
            CK(cudaMemcpyAsync(counters, std::array<uint32_t, 4>{1u, 0u, 0u, 0u}.data(), 16, cudaMemcpyHostToDevice, st));
            k_sah_root<<<grid, B, 0, st>>>(bounds, n, sah_tasks[0], pt, perm, counters + 3, bin_cap);
            ++out->kernel_launches;
            uint32_t n_tasks = 1, n_bins = 1, level = 0;
            while (n_tasks > 0) {
                uint32_t words = n_bins * SAH_TASK_WORDS;
                if (words) {
                    k_sah_init_bins<<<(words + 255) / 256, 256, 0, st>>>(sah_bins, words);
                    k_sah_bin<<<grid, B, 0, st>>>(perm, pt, n, sah_tasks[0], cen, flat, sah_bins);
                    out->kernel_launches += 2;
                }
                CK(cudaMemsetAsync(counters + 2, 0, 8, st));
                k_sah_split<<<(n_tasks + SAH_SPLIT_WARPS - 1) / SAH_SPLIT_WARPS, 32 * SAH_SPLIT_WARPS, 0, st>>>(
                    sah_tasks[0], n_tasks, sah_bins, perm, cen, flat, sah_tasks[1], counters + 2, task_cap,
                    counters + 3, bin_cap, counters, n - 1, b, level, err);
                k_sah_partition<<<grid, B, 0, st>>>(perm, pt, n, sah_tasks[0], cen, perm2, pt2);
                out->kernel_launches += 2;
                CK(cudaGetLastError());
                uint32_t hc2[2];
                CK(cudaMemcpyAsync(hc2, counters + 2, 8, cudaMemcpyDeviceToHost, st));
                CK(cudaStreamSynchronize(st));
                n_tasks = hc2[0];
                n_bins = std::min(hc2[1], bin_cap);
                std::swap(perm, perm2);
                std::swap(pt, pt2);
                std::swap(sah_tasks[0], sah_tasks[1]);
                if (n_tasks > task_cap || ++level > 4096) {
                    if (msg) *msg = "binned SAH build did not converge";
                    e = cudaErrorUnknown;
                    goto done;
                }
            }
            sv = perm;
        }
        const int width = in.width < 2 ? 2 : (in.width > 8 ? 8 : in.width);
        const uint32_t leaf_max = in.leaf_max < 1u ? 1u : (in.leaf_max > LEAF_MAX_LIMIT ? LEAF_MAX_LIMIT : in.leaf_max);
        k_refit<<<grid, B, 0, st>>>(flat, sv, (int)n, b, width, leaf_max, err);
        ++out->kernel_launches;
        CK(cudaGetLastError());
        // collapse, level by level; node 0 is the root.  The recurrence is not
        // bound to shallow trees (scenes of triangles whose sizes fall off
        // geometrically: up to 1.3 times the levels); one too deep for
        // traversal is collapsed again by opening the largest child everywhere.
        uint32_t depth = 0;
        for (uint32_t open_above : {n / 2u, 0u}) {
            const uint2 root = make_uint2(n > 1 ? 0u : LEAF, 0u);
            const uint32_t init_counts[4] = {1u, 0u, 0u, 0u};  // node alloc, tri alloc, queue out count, pad
            CK(cudaMemcpyAsync(qa, &root, sizeof(root), cudaMemcpyHostToDevice, st));
            CK(cudaMemcpyAsync(counters, init_counts, sizeof(init_counts), cudaMemcpyHostToDevice, st));
            uint32_t n_in = 1;
            depth = 0;
            out->level_start[0] = 0u;
            out->level_start[1] = 1u;
            while (n_in > 0 && depth <= 64) {
                CK(cudaMemsetAsync(counters + 2, 0, 4, st));
                k_collapse<<<(n_in + 127) / 128, 128, 0, st>>>(b, qa, n_in, qb, counters + 2, out->nodes, counters,
                                                               node_cap, out->tris, counters + 1, n, flat, sv, err,
                                                               width, leaf_max, open_above);
                ++out->kernel_launches;
                ++depth;
                CK(cudaGetLastError());
                uint32_t hc3[3];
                CK(cudaMemcpyAsync(hc3, counters, sizeof(hc3), cudaMemcpyDeviceToHost, st));
                CK(cudaStreamSynchronize(st));
                n_in = hc3[2];
                if (depth < 65) out->level_start[depth + 1] = hc3[0];  // nodes of the next level end here
                std::swap(qa, qb);
            }
            if (depth <= (uint32_t)TRAV_STACK) break;
        }
        if (depth > 64) {
            if (msg) *msg = "BVH8 collapse exceeded 64 levels";
            e = cudaErrorUnknown;
            goto done;
        }
        uint32_t hc[4], herr = 0;
        CK(cudaMemcpyAsync(hc, counters, sizeof(hc), cudaMemcpyDeviceToHost, st));
        CK(cudaMemcpyAsync(&herr, err, 4, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        if (herr & ERR_WAIT_TIMEOUT) {
            if (msg) *msg = "the sort's bounded wait gave up";
            e = cudaErrorTimeout;
            goto done;
        }
        if (herr != 0u || hc[1] != n) {
            if (msg) *msg = "BVH8 collapse produced an inconsistent tree";
            e = cudaErrorUnknown;
            goto done;
        }
        out->n_nodes = hc[0];
        out->depth = depth;
    }
done:
    out->mem = kept.detach();
    if (e != cudaSuccess) {
        cudaFree(out->mem);
        out->mem = nullptr;
        out->nodes = nullptr;
        out->tris = nullptr;
        out->tri_inst = nullptr;
        out->scatter = nullptr;
    }
#undef CK
    return e;
}

int launch_update_slots(TriSlot* tris, uint32_t n_tris, const uint32_t* tri_inst, const uint8_t* moved,
                        const float4* vtx, const uint32_t* indices, const uint4* mesh_infos, const InstDev* inst,
                        const InstFwd* fwd, cudaStream_t st) {
    if (n_tris == 0) return 0;
    k_update_slots<<<(n_tris + 255) / 256, 256, 0, st>>>(tris, n_tris, tri_inst, moved, vtx, indices, mesh_infos, inst,
                                                         fwd);
    return 1;
}

int launch_expand_lights(const LightInst* li, uint32_t n_li, const uint8_t* moved, const float4* vtx,
                         const uint32_t* indices, const uint4* mesh_infos, const InstDev* inst, const InstFwd* fwd,
                         float4* lights, cudaStream_t st) {
    if (n_li == 0) return 0;
    k_expand_lights<<<n_li, 128, 0, st>>>(li, moved, vtx, indices, mesh_infos, inst, fwd, lights);
    return 1;
}

int launch_scatter_masks(const BvhOutputs& bvh, const InstDev* inst, const float4* materials, uint8_t* mask,
                         cudaStream_t st) {
    int n = 0;
    for (int L = (int)bvh.depth - 1; L >= 0; --L) {
        const uint32_t b = bvh.level_start[L], e = bvh.level_start[L + 1];
        if (e <= b) continue;
        k_scatter_mask<<<(e - b + 127) / 128, 128, 0, st>>>(bvh.nodes, bvh.tris, bvh.tri_inst, inst, materials, b, e,
                                                            mask);
        ++n;
    }
    return n;
}

int refit_bvh8(Node8* nodes, const TriSlot* tris, const BvhOutputs& lv, float4* aux, uint32_t* err,
               cudaStream_t st) {
    int n = 0;
    for (int L = (int)lv.depth - 1; L >= 0; --L) {
        uint32_t b = lv.level_start[L], e = lv.level_start[L + 1];
        if (e <= b) continue;
        k_refit8<<<(e - b + 127) / 128, 128, 0, st>>>(nodes, tris, b, e, aux, err);
        ++n;
    }
    return n;
}

}  // namespace srt
