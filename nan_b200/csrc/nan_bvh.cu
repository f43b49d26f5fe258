// nan_bvh.cu -- GPU scene flattening and BVH construction.
//
// Replaces the reference's driver-built BLAS/TLAS (scene.py:445-533): the
// instances are flattened into one world-space triangle array (each triangle
// keeps its (instance, primitive) identity), and a binary BVH is built over
// it entirely on the GPU:
//   1. per-instance triangle counts + exclusive scan (CUB),
//   2. flatten: transform every triangle to world space, write its box,
//   3. scene bounds of the centroids (block reduction + ordered-int atomics),
//   4. 63-bit Morton codes of the centroids, radix sort (CUB),
//   5. a binary hierarchy over the sorted triangles, by one of three builders
//      (NanTuning.bvh_builder):
//      0. top-down binned SAH (k_sah_*, the default),
//      1. LBVH from the sorted codes (Karras 2012, "Maximizing parallelism in
//         the construction of BVHs, octrees, and k-d trees") with a
//         bottom-up box refit (one atomic arrival counter per node),
//      2. PLOC clustering (k_ploc_*),
//   6. for 0 and 2: SAH leaf collapse (up to 3 triangles per leaf), depth-first
//      placement and the compressed 8-wide conversion,
//   7. emission of 64-byte two-box nodes and leaf-ordered triangles.
#include <cub/cub.cuh>

#include <algorithm>
#include <cstdio>
#include <mutex>
#include <vector>

#include "nan_internal.h"

namespace {

using nan_host::cuda_fail;
using nan_host::set_error;

constexpr int kThreads = 256;

__device__ __forceinline__ uint32_t float_to_ordered(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ordered_to_float(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

__global__ void k_instance_counts(const uint4* __restrict__ instance_descs, const uint4* __restrict__ mesh_descs,
                                  uint32_t instance_count, uint32_t* __restrict__ counts) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > instance_count) return;
    if (i == instance_count) {
        counts[i] = 0u;
        return;
    }
    const uint4 id = instance_descs[i];
    counts[i] = mesh_descs[id.x].y / 3u;
}

// mul(M, float4(p, 1)).xyz, unfused, left to right (the CPU oracle's order).
__device__ __forceinline__ float3 xform(const float* __restrict__ m, float x, float y, float z) {
    return make_float3(((m[0] * x + m[1] * y) + m[2] * z) + m[3], ((m[4] * x + m[5] * y) + m[6] * z) + m[7],
                       ((m[8] * x + m[9] * y) + m[10] * z) + m[11]);
}

struct Bounds {
    uint32_t lo[3];  // ordered ints
    uint32_t hi[3];
    uint32_t max_abs;
};

__global__ void k_flatten(NanSceneDesc sd, const uint32_t* __restrict__ offsets, uint32_t tri_count,
                          float4* __restrict__ tris, uint2* __restrict__ refs, float4* __restrict__ box_lo,
                          float4* __restrict__ box_hi, Bounds* __restrict__ bounds) {
    const uint32_t f = blockIdx.x * blockDim.x + threadIdx.x;
    float c[3] = {INFINITY, INFINITY, INFINITY};
    float ch[3] = {-INFINITY, -INFINITY, -INFINITY};
    float mabs = 0.0f;
    if (f < tri_count) {
        // instance = last i with offsets[i] <= f
        uint32_t lo = 0, hi = sd.instance_count;  // search in [0, I]
        while (lo < hi) {
            const uint32_t mid = (lo + hi + 1u) >> 1;
            if (offsets[mid] <= f) lo = mid; else hi = mid - 1u;
        }
        const uint32_t inst = lo;
        const uint32_t prim = f - offsets[inst];
        const uint4 id = reinterpret_cast<const uint4*>(sd.instance_descs)[inst];
        const uint4 md = reinterpret_cast<const uint4*>(sd.mesh_descs)[id.x];
        const float* m = sd.transforms + 16u * id.z;
        float3 w[3];
        for (int k = 0; k < 3; ++k) {
            const uint32_t vi = md.z + sd.indices[md.w + 3u * prim + (uint32_t)k];
            const float* v = sd.vertices + 8u * vi;
            w[k] = xform(m, v[0], v[1], v[2]);
        }
        tris[3u * f + 0] = make_float4(w[0].x, w[0].y, w[0].z, __uint_as_float(f));
        tris[3u * f + 1] = make_float4(w[1].x, w[1].y, w[1].z, 0.0f);
        tris[3u * f + 2] = make_float4(w[2].x, w[2].y, w[2].z, 0.0f);
        refs[f] = make_uint2(inst, prim);
        float3 l = make_float3(fminf(fminf(w[0].x, w[1].x), w[2].x), fminf(fminf(w[0].y, w[1].y), w[2].y),
                               fminf(fminf(w[0].z, w[1].z), w[2].z));
        float3 h = make_float3(fmaxf(fmaxf(w[0].x, w[1].x), w[2].x), fmaxf(fmaxf(w[0].y, w[1].y), w[2].y),
                               fmaxf(fmaxf(w[0].z, w[1].z), w[2].z));
        box_lo[f] = make_float4(l.x, l.y, l.z, 0.0f);
        box_hi[f] = make_float4(h.x, h.y, h.z, 0.0f);
        c[0] = ch[0] = 0.5f * (l.x + h.x);
        c[1] = ch[1] = 0.5f * (l.y + h.y);
        c[2] = ch[2] = 0.5f * (l.z + h.z);
        mabs = fmaxf(fmaxf(fmaxf(fabsf(l.x), fabsf(h.x)), fmaxf(fabsf(l.y), fabsf(h.y))),
                     fmaxf(fabsf(l.z), fabsf(h.z)));
    }
    typedef cub::BlockReduce<float, kThreads> Reduce;
    __shared__ typename Reduce::TempStorage tmp;
    for (int a = 0; a < 3; ++a) {
        const float mn = Reduce(tmp).Reduce(c[a], cub::Min());
        __syncthreads();
        const float mx = Reduce(tmp).Reduce(ch[a], cub::Max());
        __syncthreads();
        if (threadIdx.x == 0) {
            atomicMin(&bounds->lo[a], float_to_ordered(mn));
            atomicMax(&bounds->hi[a], float_to_ordered(mx));
        }
    }
    const float ma = Reduce(tmp).Reduce(mabs, cub::Max());
    if (threadIdx.x == 0) atomicMax(&bounds->max_abs, float_to_ordered(ma));
}

__device__ __forceinline__ uint64_t expand21(uint32_t v) {
    uint64_t x = v & 0x1fffffu;
    x = (x | x << 32) & 0x1f00000000ffffull;
    x = (x | x << 16) & 0x1f0000ff0000ffull;
    x = (x | x << 8) & 0x100f00f00f00f00full;
    x = (x | x << 4) & 0x10c30c30c30c30c3ull;
    x = (x | x << 2) & 0x1249249249249249ull;
    return x;
}

__global__ void k_morton(const float4* __restrict__ box_lo, const float4* __restrict__ box_hi, uint32_t n,
                         const Bounds* __restrict__ bounds, uint64_t* __restrict__ keys, uint32_t* __restrict__ vals) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 l = box_lo[i], h = box_hi[i];
    const float c[3] = {0.5f * (l.x + h.x), 0.5f * (l.y + h.y), 0.5f * (l.z + h.z)};
    uint32_t q[3];
    for (int a = 0; a < 3; ++a) {
        const float lo = ordered_to_float(bounds->lo[a]);
        const float hi = ordered_to_float(bounds->hi[a]);
        const float ext = hi - lo;
        float u = ext > 0.0f ? (c[a] - lo) / ext : 0.0f;
        u = fminf(fmaxf(u, 0.0f), 1.0f);
        q[a] = min((uint32_t)(u * 2097152.0f), 2097151u);
    }
    keys[i] = (expand21(q[0]) << 2) | (expand21(q[1]) << 1) | expand21(q[2]);
    vals[i] = i;
}

__device__ __forceinline__ int delta(const uint64_t* __restrict__ k, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    const uint64_t a = k[i], b = k[j];
    if (a == b) return 64 + __clz((uint32_t)(i ^ j));
    return __clzll((long long)(a ^ b));
}

// Interior node i of n-1; children < n-1 are interior, leaves are encoded as
// ~leaf. parent arrays: interior parents (n-1) and leaf parents (n).
__global__ void k_hierarchy(const uint64_t* __restrict__ keys, int n, int2* __restrict__ children,
                            int* __restrict__ node_parent, int* __restrict__ leaf_parent) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    const int d = (delta(keys, n, i, i + 1) - delta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
    const int dmin = delta(keys, n, i, i - d);
    int lmax = 2;
    while (delta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
    const int j = i + l * d;
    const int dnode = delta(keys, n, i, j);
    int s = 0, t = l;
    do {
        t = (t + 1) >> 1;
        if (delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    const int gamma = i + s * d + min(d, 0);
    const int left = (min(i, j) == gamma) ? ~gamma : gamma;
    const int right = (max(i, j) == gamma + 1) ? ~(gamma + 1) : gamma + 1;
    children[i] = make_int2(left, right);
    if (left < 0) leaf_parent[~left] = i; else node_parent[left] = i;
    if (right < 0) leaf_parent[~right] = i; else node_parent[right] = i;
    if (i == 0) node_parent[0] = -1;
}

// Leaf-ordered triangles and boxes.
__global__ void k_gather_leaves(const uint32_t* __restrict__ order, uint32_t n, const float4* __restrict__ tris_flat,
                                const float4* __restrict__ lo_flat, const float4* __restrict__ hi_flat,
                                float4* __restrict__ tris, float4* __restrict__ leaf_lo, float4* __restrict__ leaf_hi) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t f = order[i];
    tris[3u * i + 0] = tris_flat[3u * f + 0];
    tris[3u * i + 1] = tris_flat[3u * f + 1];
    tris[3u * i + 2] = tris_flat[3u * f + 2];
    leaf_lo[i] = lo_flat[f];
    leaf_hi[i] = hi_flat[f];
}

__device__ __forceinline__ void child_box(int c, const float4* node_lo, const float4* node_hi, const float4* leaf_lo,
                                          const float4* leaf_hi, float4* lo, float4* hi) {
    if (c < 0) {
        *lo = leaf_lo[~c];
        *hi = leaf_hi[~c];
    } else {
        *lo = __ldcg(node_lo + c);
        *hi = __ldcg(node_hi + c);
    }
}

// Every walk from a leaf or node up to the root stops after kMaxWalk steps
// or at a parent index outside [0, interior): a malformed hierarchy then
// yields a depth above the traversal stack's (rejected by the host) instead of
// a walk that never ends. Valid trees have depth <= 96 here.
constexpr uint32_t kMaxWalk = 4096u;
__device__ __forceinline__ bool walk_on(int p, uint32_t interior, uint32_t steps) {
    return p >= 0 && (uint32_t)p < interior && steps < kMaxWalk;
}

// Bottom-up refit: the second thread to reach a node computes its box.
__global__ void k_refit(uint32_t n, const int2* __restrict__ children, const int* __restrict__ node_parent,
                        const int* __restrict__ leaf_parent, const float4* __restrict__ leaf_lo,
                        const float4* __restrict__ leaf_hi, float4* node_lo, float4* node_hi,
                        uint32_t* __restrict__ arrivals) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int p = leaf_parent[i];
    for (uint32_t steps = 0; walk_on(p, n - 1u, steps); ++steps) {
        __threadfence();
        if (atomicAdd(&arrivals[p], 1u) == 0u) return;
        const int2 ch = children[p];
        float4 al, ah, bl, bh;
        child_box(ch.x, node_lo, node_hi, leaf_lo, leaf_hi, &al, &ah);
        child_box(ch.y, node_lo, node_hi, leaf_lo, leaf_hi, &bl, &bh);
        __stcg(node_lo + p, make_float4(fminf(al.x, bl.x), fminf(al.y, bl.y), fminf(al.z, bl.z), 0.0f));
        __stcg(node_hi + p, make_float4(fmaxf(ah.x, bh.x), fmaxf(ah.y, bh.y), fmaxf(ah.z, bh.z), 0.0f));
        p = node_parent[p];
    }
}

// Depth of every leaf (steps to the root); max over leaves is the tree depth.
__global__ void k_depth(uint32_t n, const int* __restrict__ node_parent, const int* __restrict__ leaf_parent,
                        uint32_t* __restrict__ max_depth) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t depth = 1;
    int p = leaf_parent[i];
    while (walk_on(p, n - 1u, depth)) {
        ++depth;
        p = node_parent[p];
    }
    if (p >= 0) depth = kMaxWalk;  // a parent out of range or a walk too long: reject
    atomicMax(max_depth, depth);
}

__device__ __forceinline__ float half_area(float4 l, float4 h) {
    const float x = h.x - l.x, y = h.y - l.y, z = h.z - l.z;
    return x * y + y * z + z * x;
}

// 64-byte nodes with padded child boxes; also accumulates the SAH cost.
// Adds each lane's SAH term into *sah with one atomic per warp (a single
// address takes one atomic per node otherwise, which serialises millions of
// them). Every lane of the warp must call it.
__device__ __forceinline__ void add_sah(double* sah, double cost) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cost += __shfl_down_sync(0xffffffffu, cost, o);
    if ((threadIdx.x & 31u) == 0u && cost != 0.0) atomicAdd(sah, cost);
}

// Outward padding of the binary node boxes: 1.5 x 2^-18 of the scene's
// largest coordinate M. The slab test (box2 in nan_scene.cuh) rounds
// distances that reach |o| + M along an axis at most four times, 4 x 2^-24 of
// them, so it never culls a box the exact ray crosses while the ray's origin
// lies within about 20 M.
__device__ __forceinline__ float node_pad(const Bounds* bounds) {
    return ordered_to_float(bounds->max_abs) * 5.7220458984375e-6f + 1e-30f;
}

// Padded interval [lo - pad, hi + pad] as (centre, half extent), the half
// extent rounded up so that the centre's rounding never shrinks the interval.
// A half extent above kOpenExtent (or a NaN) leaves the interval open, as
// (0, infinity): with reciprocals of up to 1e20 (box_setup) the centre's
// product overflows for a ray well inside such an interval, and an infinite
// near distance would cull it.
constexpr float kOpenExtent = 1e18f;

__device__ __forceinline__ float2 centre_half(float lo, float hi, float pad) {
    const float l = lo - pad, h = hi + pad;
    const float c = 0.5f * l + 0.5f * h;
    const float e = fmaxf(__fsub_ru(h, c), __fsub_ru(c, l));
    return e <= kOpenExtent ? make_float2(c, e) : make_float2(0.0f, INFINITY);
}

// The three box words of a binary node (layout: SceneView, nan_scene.cuh).
__device__ __forceinline__ void store_node_boxes(float4* node, float4 al, float4 ah, float4 bl, float4 bh, float pad) {
    const float2 ax = centre_half(al.x, ah.x, pad), bx = centre_half(bl.x, bh.x, pad);
    const float2 ay = centre_half(al.y, ah.y, pad), by = centre_half(bl.y, bh.y, pad);
    const float2 az = centre_half(al.z, ah.z, pad), bz = centre_half(bl.z, bh.z, pad);
    node[0] = make_float4(ax.x, bx.x, ay.x, by.x);
    node[1] = make_float4(az.x, bz.x, ax.y, bx.y);
    node[2] = make_float4(ay.y, by.y, az.y, bz.y);
}

__global__ void k_emit(uint32_t interior, const int2* __restrict__ children, const float4* __restrict__ node_lo,
                       const float4* __restrict__ node_hi, const float4* __restrict__ leaf_lo,
                       const float4* __restrict__ leaf_hi, const Bounds* __restrict__ bounds,
                       float4* __restrict__ nodes, double* __restrict__ sah) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    double cost = 0.0;
    if (i < interior) {
        const float pad = node_pad(bounds);
        const int2 ch = children[i];
        float4 al, ah, bl, bh;
        child_box(ch.x, node_lo, node_hi, leaf_lo, leaf_hi, &al, &ah);
        child_box(ch.y, node_lo, node_hi, leaf_lo, leaf_hi, &bl, &bh);
        store_node_boxes(nodes + 4u * i, al, ah, bl, bh, pad);
        // leaves (single triangles in LBVH) as ~(first << 3 | count - 1)
        const int rx = ch.x < 0 ? ~((~ch.x) << 3) : ch.x;
        const int ry = ch.y < 0 ? ~((~ch.y) << 3) : ch.y;
        nodes[4u * i + 3] = make_float4(__int_as_float(rx), __int_as_float(ry), 0.0f, 0.0f);
        const float root_area = fmaxf(half_area(node_lo[0], node_hi[0]), 1e-30f);
        cost = (double)(half_area(node_lo[i], node_hi[i]) / root_area);  // one traversal step
        if (ch.x < 0) cost += (double)(half_area(al, ah) / root_area);   // one triangle per leaf
        if (ch.y < 0) cost += (double)(half_area(bl, bh) / root_area);
    }
    add_sah(sah, cost);
}


// ---------------------------------------------------------------------------
// PLOC: parallel locally-ordered clustering (Meister and Bittner 2018).
// Clusters start as the Morton-sorted triangles; every iteration each cluster
// finds the neighbour within +-kPlocRadius positions whose union box has the
// smallest surface area, mutual nearest neighbours merge into a new interior
// node, and the cluster list is compacted (order preserved).
// ---------------------------------------------------------------------------
constexpr int kPlocRadius = 64;
constexpr int kPlocBlock = 256;
constexpr int kPlocBatch = 8;       // PLOC iterations between two host checks of the count
constexpr int kWideBatch = 4;       // wide-conversion levels between two host checks
constexpr int kWideMaxLevels = 256;
constexpr int kMaxLeafTris = 3;  // the wide nodes' leaf encoding holds up to 3 triangles

__device__ __forceinline__ float area_union(float4 al, float4 ah, float4 bl, float4 bh) {
    const float x = fmaxf(ah.x, bh.x) - fminf(al.x, bl.x);
    const float y = fmaxf(ah.y, bh.y) - fminf(al.y, bl.y);
    const float z = fmaxf(ah.z, bh.z) - fminf(al.z, bl.z);
    return x * y + y * z + z * x;
}

__global__ void k_ploc_init(uint32_t n, int* __restrict__ idx) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) idx[i] = ~(int)i;
}

// The PLOC kernels read the current cluster count from device memory
// (*count), so that several iterations run back to back without the host;
// grids are sized for an upper bound of the count, and with one cluster left
// every kernel does nothing.
__global__ void __launch_bounds__(kPlocBlock) k_ploc_nn(const uint32_t* __restrict__ count,
                                                         const float4* __restrict__ lo,
                                                         const float4* __restrict__ hi, int* __restrict__ nn) {
    const int c = (int)*count;
    if (c <= 1) return;
    __shared__ float4 slo[kPlocBlock + 2 * kPlocRadius];
    __shared__ float4 shi[kPlocBlock + 2 * kPlocRadius];
    const int b0 = blockIdx.x * kPlocBlock;
    for (int k = threadIdx.x; k < kPlocBlock + 2 * kPlocRadius; k += blockDim.x) {
        const int g = b0 - kPlocRadius + k;
        if (g >= 0 && g < c) {
            slo[k] = lo[g];
            shi[k] = hi[g];
        }
    }
    __syncthreads();
    const int i = b0 + (int)threadIdx.x;
    if (i >= c) return;
    const float4 ml = slo[threadIdx.x + kPlocRadius], mh = shi[threadIdx.x + kPlocRadius];
    float best = INFINITY;
    int bj = -1;
    for (int dj = -kPlocRadius; dj <= kPlocRadius; ++dj) {
        const int j = i + dj;
        if (dj == 0 || j < 0 || j >= c) continue;
        const float a = area_union(ml, mh, slo[threadIdx.x + kPlocRadius + dj], shi[threadIdx.x + kPlocRadius + dj]);
        if (a < best) {  // ties keep the lower index (dj ascending)
            best = a;
            bj = j;
        }
    }
    nn[i] = bj;
}

// Also clears valid[c .. bound] (bound + 1 flags are scanned).
__global__ void k_ploc_merge(const uint32_t* __restrict__ count, int bound, const int* __restrict__ nn,
                             const int* __restrict__ idx,
                             const float4* __restrict__ lo, const float4* __restrict__ hi, int* __restrict__ idx2,
                             float4* __restrict__ lo2, float4* __restrict__ hi2, uint32_t* __restrict__ valid,
                             int2* __restrict__ children, int* __restrict__ node_parent, int* __restrict__ leaf_parent,
                             float4* __restrict__ node_lo, float4* __restrict__ node_hi, uint32_t* node_counter) {
    const int c = (int)*count;
    if (c <= 1) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > bound) return;
    if (i >= c) {
        valid[i] = 0u;
        return;
    }
    const int j = nn[i];
    if (j >= 0 && nn[j] == i) {
        if (i > j) {
            valid[i] = 0u;
            return;
        }
        const int id = (int)atomicAdd(node_counter, 1u);
        const int a = idx[i], b = idx[j];
        const float4 al = lo[i], ah = hi[i], bl = lo[j], bh = hi[j];
        const float4 l = make_float4(fminf(al.x, bl.x), fminf(al.y, bl.y), fminf(al.z, bl.z), 0.0f);
        const float4 h = make_float4(fmaxf(ah.x, bh.x), fmaxf(ah.y, bh.y), fmaxf(ah.z, bh.z), 0.0f);
        children[id] = make_int2(a, b);
        if (a < 0) leaf_parent[~a] = id; else node_parent[a] = id;
        if (b < 0) leaf_parent[~b] = id; else node_parent[b] = id;
        node_lo[id] = l;
        node_hi[id] = h;
        idx2[i] = id;
        lo2[i] = l;
        hi2[i] = h;
    } else {
        idx2[i] = idx[i];
        lo2[i] = lo[i];
        hi2[i] = hi[i];
    }
    valid[i] = 1u;
}

// Also writes the next iteration's count (the kept clusters) to *next_count:
// the count is double-buffered, iteration k reading slot k & 1.
__global__ void k_ploc_compact(const uint32_t* __restrict__ count, uint32_t* __restrict__ next_count,
                               const uint32_t* __restrict__ valid, const uint32_t* __restrict__ pos,
                               const int* __restrict__ idx2, const float4* __restrict__ lo2,
                               const float4* __restrict__ hi2, int* __restrict__ idx, float4* __restrict__ lo,
                               float4* __restrict__ hi) {
    const int c = (int)*count;
    if (blockIdx.x == 0 && threadIdx.x == 0) *next_count = c <= 1 ? (uint32_t)c : pos[c];
    if (c <= 1) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c || !valid[i]) return;
    const uint32_t p = pos[i];
    idx[p] = idx2[i];
    lo[p] = lo2[i];
    hi[p] = hi2[i];
}

__device__ __forceinline__ float half_area4(float4 l, float4 h) {
    const float x = h.x - l.x, y = h.y - l.y, z = h.z - l.z;
    return x * y + y * z + z * x;
}

// Bottom-up: triangle count, kept-interior count and SAH cost (relative to
// the node's own area, C_trav = C_int = 1) of every subtree; a subtree of at
// most kMaxLeafTris triangles collapses into one leaf when that is cheaper.
struct SubtreeInfo {
    uint32_t tris;
    uint32_t interior;  // kept interior nodes (0 when collapsed)
    float cost;
    uint32_t collapsed;
};

__device__ __forceinline__ void child_info(int c, const SubtreeInfo* info, uint32_t* tris, uint32_t* interior,
                                           float* cost) {
    if (c < 0) {
        *tris = 1u;
        *interior = 0u;
        *cost = 1.0f;
    } else {
        const volatile SubtreeInfo* v = info + c;  // written by the sibling's thread
        *tris = v->tris;
        *interior = v->interior;
        *cost = v->cost;
    }
}

__global__ void k_subtree(uint32_t n, const int2* __restrict__ children, const int* __restrict__ node_parent,
                          const int* __restrict__ leaf_parent, const float4* __restrict__ leaf_lo,
                          const float4* __restrict__ leaf_hi, const float4* __restrict__ node_lo,
                          const float4* __restrict__ node_hi, SubtreeInfo* info, uint32_t* __restrict__ arrivals) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int p = leaf_parent[i];
    for (uint32_t steps = 0; walk_on(p, n - 1u, steps); ++steps) {
        __threadfence();
        if (atomicAdd(&arrivals[p], 1u) == 0u) return;
        const int2 ch = children[p];
        uint32_t ta, ia, tb, ib;
        float ca, cb;
        child_info(ch.x, info, &ta, &ia, &ca);
        child_info(ch.y, info, &tb, &ib, &cb);
        const float ap = fmaxf(half_area4(node_lo[p], node_hi[p]), 1e-30f);
        const float aa = ch.x < 0 ? half_area4(leaf_lo[~ch.x], leaf_hi[~ch.x]) : half_area4(node_lo[ch.x], node_hi[ch.x]);
        const float ab = ch.y < 0 ? half_area4(leaf_lo[~ch.y], leaf_hi[~ch.y]) : half_area4(node_lo[ch.y], node_hi[ch.y]);
        const float split = 1.0f + (aa * ca + ab * cb) / ap;
        const uint32_t tris = ta + tb;
        SubtreeInfo v;
        v.tris = tris;
        if (tris <= (uint32_t)kMaxLeafTris && (float)tris <= split) {
            v.cost = (float)tris;
            v.interior = 0u;
            v.collapsed = 1u;
        } else {
            v.cost = split;
            v.interior = 1u + ia + ib;
            v.collapsed = 0u;
        }
        volatile SubtreeInfo* dst = info + p;
        dst->tris = v.tris;
        dst->interior = v.interior;
        dst->cost = v.cost;
        dst->collapsed = v.collapsed;
        p = node_parent[p];
    }
}

// Depth-first placement: walking up from a node or triangle to the root,
// every step from a right child skips the left sibling's interior nodes (for
// the node index) or triangles (for the triangle position). Nodes below a
// collapsed ancestor are not emitted (dfs = -1).
__global__ void k_dfs_nodes(uint32_t interior, const int2* __restrict__ children, const int* __restrict__ node_parent,
                            const SubtreeInfo* __restrict__ info, int* __restrict__ dfs, uint32_t* __restrict__ tri_off) {
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= interior) return;
    int node = (int)x;
    int index = 0;
    uint32_t toff = 0u;
    bool hidden = false;
    int p = node_parent[node];
    for (uint32_t steps = 0; walk_on(p, interior, steps); ++steps) {
        const SubtreeInfo pi = info[p];
        if (pi.collapsed) hidden = true;
        const int2 ch = children[p];
        index += 1;
        if (ch.y == node) {
            if (ch.x >= 0) {
                const SubtreeInfo li = info[ch.x];
                index += (int)li.interior;
                toff += li.tris;
            } else {
                toff += 1u;
            }
        }
        node = p;
        p = node_parent[p];
    }
    dfs[x] = hidden ? -1 : index;
    tri_off[x] = toff;
}

__global__ void k_dfs_leaves(uint32_t n, const int2* __restrict__ children, const int* __restrict__ node_parent,
                             const int* __restrict__ leaf_parent, const SubtreeInfo* __restrict__ info,
                             uint32_t* __restrict__ tri_pos) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int node = ~(int)i;
    uint32_t toff = 0u;
    int p = leaf_parent[i];
    for (uint32_t steps = 0; walk_on(p, n - 1u, steps); ++steps) {
        const int2 ch = children[p];
        if (ch.y == node) toff += ch.x >= 0 ? info[ch.x].tris : 1u;
        node = p;
        p = node_parent[p];
    }
    tri_pos[i] = toff;
}

__global__ void k_scatter_tris(uint32_t n, const uint32_t* __restrict__ tri_pos, const float4* __restrict__ src,
                               float4* __restrict__ dst) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t p = tri_pos[i];
    dst[3u * p] = src[3u * i];
    dst[3u * p + 1] = src[3u * i + 1];
    dst[3u * p + 2] = src[3u * i + 2];
}

__device__ __forceinline__ int child_ref(int c, const int* dfs, const uint32_t* tri_off, const uint32_t* tri_pos,
                                         const SubtreeInfo* info) {
    if (c < 0) return ~(int)(tri_pos[~c] << 3);
    const SubtreeInfo v = info[c];
    if (v.collapsed) return ~(int)((tri_off[c] << 3) | (v.tris - 1u));
    return dfs[c];
}

__global__ void k_emit_dfs(uint32_t interior, const int2* __restrict__ children, const float4* __restrict__ node_lo,
                           const float4* __restrict__ node_hi, const float4* __restrict__ leaf_lo,
                           const float4* __restrict__ leaf_hi, const Bounds* __restrict__ bounds,
                           const SubtreeInfo* __restrict__ info, const int* __restrict__ dfs,
                           const uint32_t* __restrict__ tri_off, const uint32_t* __restrict__ tri_pos, int root,
                           float4* __restrict__ nodes, double* __restrict__ sah) {
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
    const int slot = x < interior ? dfs[x] : -1;
    double cost = 0.0;
    if (slot >= 0 && !info[x].collapsed) {
        const float pad = node_pad(bounds);
        const int2 ch = children[x];
        float4 al, ah, bl, bh;
        child_box(ch.x, node_lo, node_hi, leaf_lo, leaf_hi, &al, &ah);
        child_box(ch.y, node_lo, node_hi, leaf_lo, leaf_hi, &bl, &bh);
        store_node_boxes(nodes + 4u * slot, al, ah, bl, bh, pad);
        const int ra = child_ref(ch.x, dfs, tri_off, tri_pos, info);
        const int rb = child_ref(ch.y, dfs, tri_off, tri_pos, info);
        nodes[4u * slot + 3] = make_float4(__int_as_float(ra), __int_as_float(rb), 0.0f, 0.0f);
        const float root_area = fmaxf(half_area4(node_lo[root], node_hi[root]), 1e-30f);
        cost = (double)(half_area4(node_lo[x], node_hi[x]) / root_area);
        if (ra < 0) cost += (double)(half_area4(al, ah) / root_area) * (double)(((~ra) & 7) + 1);
        if (rb < 0) cost += (double)(half_area4(bl, bh) / root_area) * (double)(((~rb) & 7) + 1);
    }
    add_sah(sah, cost);
}


// ---------------------------------------------------------------------------
// Compressed 8-wide BVH (after Ylitie, Karras and Laine, "Efficient Incoherent
// Ray Traversal on GPUs Through Compressed Wide BVHs", HPG 2017), converted
// top-down from the collapsed binary tree (binned SAH or PLOC): each wide
// node takes up to 8 subtrees by repeatedly opening the largest-area interior
// binary node, places them in slots ordered by octant direction, stores its
// interior children
// contiguously (child_base) and its leaf triangles contiguously (tri_base),
// and quantizes the children's boxes to 8 bits against the node's box.
// Node (80 B): w0 = (p.xyz, e.x | e.y << 8 | e.z << 16 | imask << 24)
//              w1 = (child_base, tri_base, meta[0..3], meta[4..7])
//              w2..w4 = qlo.x, qlo.y, qlo.z, qhi.x, qhi.y, qhi.z (8 bytes each)
// meta[slot]: 0 empty; interior slots are marked in imask; a leaf slot holds
// (unary triangle count) << 5 | (triangle offset from tri_base).
// ---------------------------------------------------------------------------
struct WideItem {
    int bnode;      // binary node (>= 0) or leaf code (~sorted leaf)
    uint32_t wnode;
};

__device__ __forceinline__ bool expandable(int c, const SubtreeInfo* info) { return c >= 0 && !info[c].collapsed; }

__device__ __forceinline__ void entry_box(int c, const float4* node_lo, const float4* node_hi, const float4* leaf_lo,
                                          const float4* leaf_hi, float4* lo, float4* hi) {
    if (c < 0) {
        *lo = leaf_lo[~c];
        *hi = leaf_hi[~c];
    } else {
        *lo = node_lo[c];
        *hi = node_hi[c];
    }
}

// The first level of the wide conversion: the binary root (the last cluster).
__global__ void k_wide_root(const int* __restrict__ root, WideItem* __restrict__ items) {
    items[0] = WideItem{root[0], 0u};
}

// One level of the wide conversion: *count_in items of this level in, the
// next level's items appended at *count_out (counters[0] and [1] count the
// wide nodes and triangles written so far). Eight lanes take a node: a lane
// holds an entry while the node opens, then the child of its slot. Space for
// the children is taken from the counters once a block. With one thread a node
// the entries, scores and bytes lay in local memory and every node queued at
// the counters: 200k triangles,
// 8 levels, 532 us; 143 us in this form.
constexpr int kWideLanes = 8;

__global__ void __launch_bounds__(kThreads) k_wide_level(
    const WideItem* __restrict__ items, const uint32_t* __restrict__ count_in, WideItem* __restrict__ items_out,
    uint32_t* __restrict__ count_out, uint32_t* __restrict__ counters, const int2* __restrict__ children,
    const float4* __restrict__ node_lo, const float4* __restrict__ node_hi, const float4* __restrict__ leaf_lo,
    const float4* __restrict__ leaf_hi, const SubtreeInfo* __restrict__ info, const uint32_t* __restrict__ tri_off,
    const uint32_t* __restrict__ tri_pos, const float4* __restrict__ tris_dfs, const Bounds* __restrict__ bounds,
    uint4* __restrict__ wnodes, float4* __restrict__ wtris) {
    constexpr uint32_t kFull = 0xffffffffu;
    __shared__ uint32_t s_count[2], s_base[3];
    const uint32_t count = *count_in;
    if ((uint64_t)blockIdx.x * (kThreads / kWideLanes) >= count) return;  // the whole block
    if (threadIdx.x < 2) s_count[threadIdx.x] = 0u;
    const uint32_t lane = threadIdx.x & 31u, sl = lane & 7u, group = lane & 24u;
    const uint32_t k = blockIdx.x * (kThreads / kWideLanes) + threadIdx.x / kWideLanes;
    const bool live = k < count;
    const WideItem it = live ? items[k] : WideItem{0, 0u};
    // entries: lane i of the group holds entry i < m
    int ent = 0;
    bool inner = false;  // the entry can be opened
    float4 lo = make_float4(0.0f, 0.0f, 0.0f, 0.0f), hi = lo;
    auto take = [&](int c) {
        ent = c;
        inner = expandable(c, info);
        entry_box(c, node_lo, node_hi, leaf_lo, leaf_hi, &lo, &hi);
    };
    uint32_t m = 0u;
    if (live) {
        if (expandable(it.bnode, info)) {
            const int2 ch = children[it.bnode];
            if (sl < 2u) take(sl ? ch.y : ch.x);
            m = 2u;
        } else {  // a root that is a single leaf
            if (sl == 0u) take(it.bnode);
            m = 1u;
        }
    }
    // open the largest entry (the first of equals) while there is room
    for (int step = 0; step < kWideLanes - 1; ++step) {
        float area = -1.0f;
        if (sl < m && inner) {
            const float x = half_area4(lo, hi);
            area = x > -1.0f ? x : -1.0f;
        }
        float most = area;
#pragma unroll
        for (int d = 1; d < kWideLanes; d <<= 1) most = fmaxf(most, __shfl_xor_sync(kFull, most, d));
        const uint32_t hits = (__ballot_sync(kFull, area == most) >> group) & 0xffu;
        const uint32_t best = (uint32_t)__ffs(hits) - 1u;
        const bool open = live && m < (uint32_t)kWideLanes && most > -1.0f;
        if (__ballot_sync(kFull, open) == 0u) break;
        int2 ch = make_int2(0, 0);
        if (open && sl == best) ch = children[ent];
        const int second = __shfl_sync(kFull, ch.y, (int)(group + (best & 7u)));
        if (open) {
            if (sl == best) take(ch.x);
            else if (sl == m) take(second);
            ++m;
        }
    }
    // node box, over the entries in order
    float4 plo = lo, phi = hi;
    {
        const bool has = sl < m;
        float v[6] = {has ? lo.x : INFINITY, has ? lo.y : INFINITY, has ? lo.z : INFINITY,
                      has ? -hi.x : INFINITY, has ? -hi.y : INFINITY, has ? -hi.z : INFINITY};
#pragma unroll
        for (int d = 1; d < kWideLanes; d <<= 1)
#pragma unroll
            for (int q = 0; q < 6; ++q) v[q] = fminf(v[q], __shfl_xor_sync(kFull, v[q], d));
        plo = make_float4(v[0], v[1], v[2], 0.0f);
        phi = make_float4(-v[3], -v[4], -v[5], 0.0f);
    }
    // slots by octant direction of each entry's centre: the best (entry, slot)
    // pair left, the first of equals, m times; lane `slot` notes its entry
    const float vx = 0.5f * (lo.x + hi.x) - 0.5f * (plo.x + phi.x);
    const float vy = 0.5f * (lo.y + hi.y) - 0.5f * (plo.y + phi.y);
    const float vz = 0.5f * (lo.z + hi.z) - 0.5f * (plo.z + phi.z);
    uint32_t free_slots = 0xffu;
    bool placed = !(sl < m);
    int entry_of = -1;
    for (int r = 0; r < kWideLanes; ++r) {
        const bool more = (uint32_t)r < m;
        if (__ballot_sync(kFull, more) == 0u) break;
        float score = -INFINITY;
        uint32_t slot = (uint32_t)__ffs(free_slots) - 1u;
        bool first = true;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float x = ((q & 1) ? vx : -vx) + ((q & 2) ? vy : -vy) + ((q & 4) ? vz : -vz);
            if (((free_slots >> q) & 1u) && (first || x > score)) {
                score = x;
                slot = (uint32_t)q;
                first = false;
            }
        }
        // a NaN score counts as the lowest
        const float mine = placed || !(score == score) ? -INFINITY : score;
        float most = mine;
#pragma unroll
        for (int d = 1; d < kWideLanes; d <<= 1) most = fmaxf(most, __shfl_xor_sync(kFull, most, d));
        const uint32_t hits = (__ballot_sync(kFull, !placed && mine == most) >> group) & 0xffu;
        const uint32_t who = hits ? (uint32_t)__ffs(hits) - 1u : 0u;
        const uint32_t to = __shfl_sync(kFull, slot, (int)(group + who));
        if (more) {
            if (sl == who) placed = true;
            if (sl == to) entry_of = (int)who;
            free_slots &= ~(1u << to);
        }
    }
    // each lane's slot: its child's code, box and kind
    const int from = (int)group + max(entry_of, 0);
    const int child = __shfl_sync(kFull, ent, from);
    const bool filled = entry_of >= 0;
    const bool is_inner = (__shfl_sync(kFull, inner ? 1 : 0, from) != 0) && filled;
    const float clo[3] = {__shfl_sync(kFull, lo.x, from), __shfl_sync(kFull, lo.y, from),
                          __shfl_sync(kFull, lo.z, from)};
    const float chi[3] = {__shfl_sync(kFull, hi.x, from), __shfl_sync(kFull, hi.y, from),
                          __shfl_sync(kFull, hi.z, from)};
    // allocation: interior children and leaf triangles, both in slot order
    const uint32_t imask = (__ballot_sync(kFull, is_inner) >> group) & 0xffu;
    const uint32_t rank = (uint32_t)__popc(imask & ((1u << sl) - 1u)), n_int = (uint32_t)__popc(imask);
    const uint32_t tris = !filled || is_inner ? 0u : child < 0 ? 1u : info[child].tris;
    uint32_t toff = tris;
#pragma unroll
    for (uint32_t d = 1u; d < (uint32_t)kWideLanes; d <<= 1) {
        const uint32_t up = __shfl_up_sync(kFull, toff, d, kWideLanes);
        if (sl >= d) toff += up;
    }
    const uint32_t n_tri = __shfl_sync(kFull, toff, (int)group + 7);
    toff -= tris;
    __syncthreads();
    uint32_t at_int = 0u, at_tri = 0u;
    if (sl == 0u) {
        at_int = n_int ? atomicAdd(&s_count[0], n_int) : 0u;
        at_tri = n_tri ? atomicAdd(&s_count[1], n_tri) : 0u;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t ints = s_count[0], all = s_count[1];
        s_base[0] = ints ? atomicAdd(&counters[0], ints) : 0u;
        s_base[1] = all ? atomicAdd(&counters[1], all) : 0u;
        s_base[2] = ints ? atomicAdd(count_out, ints) : 0u;
    }
    __syncthreads();
    at_int = __shfl_sync(kFull, at_int, (int)group);
    at_tri = __shfl_sync(kFull, at_tri, (int)group);
    const uint32_t child_base = s_base[0] + at_int, tri_base = s_base[1] + at_tri, out_base = s_base[2] + at_int;
    // quantization grid: p = node lo, scale 2^e with 255 * 2^e >= extent; lane
    // a finds axis a's
    const float pad = ordered_to_float(bounds->max_abs) * 3.814697265625e-6f + 1e-30f;
    const double alo = (double)(sl == 0u ? plo.x : sl == 1u ? plo.y : plo.z) - pad;
    const double ahi = (double)(sl == 0u ? phi.x : sl == 1u ? phi.y : phi.z) + pad;
    float p = (float)alo;
    if ((double)p > alo) p = nextafterf(p, -INFINITY);  // p <= lo
    const double ext = ahi - (double)p;
    int e = -126;
    if (ext > 0.0) {
        e = (int)ceil(log2(ext / 255.0));
        while (ldexp(255.0, e) < ext) ++e;
        e = max(min(e, 127), -126);
    }
    // the child's box on the grid (a scale of 2^e divides exactly); empty slots
    // hold an inverted box
    uint32_t quant[6];
    float p3[3];
    uint32_t ebits = 0u;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        p3[a] = __shfl_sync(kFull, p, (int)group + a);
        const int ea = __shfl_sync(kFull, e, (int)group + a);
        ebits |= (uint32_t)(ea + 127) << (8 * a);
        const double inv = __longlong_as_double((long long)(1023 - ea) << 52);
        const double ql = floor((((double)clo[a] - pad) - (double)p3[a]) * inv);
        const double qh = ceil((((double)chi[a] + pad) - (double)p3[a]) * inv);
        quant[a] = filled ? (uint32_t)(uint8_t)fmax(0.0, fmin(255.0, ql)) : 1u;
        quant[3 + a] = filled ? (uint32_t)(uint8_t)fmax(0.0, fmin(255.0, qh)) : 0u;
    }
    uint32_t meta = 0u;
    if (live && filled) {
        if (is_inner) {
            items_out[out_base + rank] = WideItem{child, child_base + rank};
        } else {
            const uint32_t src = child < 0 ? tri_pos[~child] : tri_off[child];
            for (uint32_t t = 0; t < tris; ++t) {
                const uint32_t d = tri_base + toff + t;
                wtris[3u * d + 0] = tris_dfs[3u * (src + t) + 0];
                wtris[3u * d + 1] = tris_dfs[3u * (src + t) + 1];
                wtris[3u * d + 2] = tris_dfs[3u * (src + t) + 2];
            }
            meta = ((tris == 1u ? 1u : (tris == 2u ? 3u : 7u)) << 5) | toff;
        }
    }
    // four lanes' bytes make a word
    uint32_t* w = reinterpret_cast<uint32_t*>(wnodes + 5u * (size_t)it.wnode);
    auto word = [&](uint32_t v) {
        v <<= 8u * (sl & 3u);
        v |= __shfl_xor_sync(kFull, v, 1);
        return v | __shfl_xor_sync(kFull, v, 2);
    };
    const uint32_t metas = word(meta);
    uint32_t quants[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) quants[q] = word(quant[q]);
    if (!live || (sl & 3u) != 0u) return;
    const uint32_t half = sl >> 2;
    if (half == 0u) {
        *reinterpret_cast<uint4*>(w) = make_uint4(__float_as_uint(p3[0]), __float_as_uint(p3[1]),
                                                  __float_as_uint(p3[2]), ebits | (imask << 24));
        *reinterpret_cast<uint2*>(w + 4) = make_uint2(child_base, tri_base);
    }
    w[6u + half] = metas;
#pragma unroll
    for (int q = 0; q < 6; ++q) w[8u + 2u * (uint32_t)q + half] = quants[q];
}

// ---------------------------------------------------------------------------
// Top-down binned SAH (Wald, "On fast construction of SAH-based bounding
// volume hierarchies", 2007): every node bins its triangles' centroids into
// kSahBins equal intervals of the node's centroid bounds on each axis and
// splits at the bin boundary of least (left area x left count + right area x
// right count), down to single triangles; the SAH leaf collapse and the
// depth-first emission above then run on this tree as on PLOC's.
// Nodes of more than kSahMidMax triangles are split level by level over the
// whole GPU: bins accumulate in shared memory by block, then with atomics, a
// warp per node picks the split, and a scan of the left flags partitions each
// node's range stably. A block builds each node of at most kSahMidMax
// triangles down to kSahSeqMax, and a warp each node of at most kSahSeqMax,
// with the same split rule.
// A node whose centroids coincide on every axis splits its range in half.
// ---------------------------------------------------------------------------
constexpr int kSahBins = 32;
constexpr uint32_t kSahSeqMax = 64;
constexpr uint32_t kSahMidMax = 1024;
constexpr int kSahBinWords = 13;  // box lo, hi, centroid lo, hi (ordered ints), count
constexpr int kSahTaskWords = 3 * kSahBins * kSahBinWords;
constexpr int kSahMaxLevels = 512;
constexpr int kSahBatch = 2;

struct SahTask {
    uint32_t first, count;
    int node;
    int axis;           // split axis, -1: halve the range
    uint32_t clo[3], chi[3];  // centroid bounds (ordered ints)
    uint32_t split_bin;       // bins <= split_bin go left
    uint32_t left_count;
    int child_task[2];  // next-level large task, or -1
};

struct SahSmall {
    uint32_t first, count;
    int node;
};

// interior nodes allocated, large tasks of the next level (appended), small
// tasks (appended), large tasks of the current level
struct SahCounters {
    uint32_t nodes, large, small, level;
    uint32_t overflow;  // nonzero: a bound below was exceeded (nothing was written past it)
    uint32_t mid;       // mid tasks (appended)
};

// Capacities of the next-level task list, the small-task list, the interior
// nodes (n - 1) and the mid-task list.
struct SahLimits {
    uint32_t large, small, nodes, mid;
};

__device__ __forceinline__ float sah_half_area(float lx, float ly, float lz, float hx, float hy, float hz) {
    const float dx = hx - lx, dy = hy - ly, dz = hz - lz;
    if (!(dx >= 0.0f)) return 0.0f;  // empty box
    return dx * dy + dy * dz + dz * dx;
}

// Bin of centroid c on an axis with centroid bounds [lo, hi]; every centroid
// lands in bin 0 when the bounds have no extent.
__device__ __forceinline__ int sah_bin(float c, float lo, float hi) {
    const float ext = hi - lo;
    if (!(ext > 0.0f)) return 0;
    const float scale = (float)kSahBins / ext;
    const int b = (int)((c - lo) * scale);
    return min(max(b, 0), kSahBins - 1);
}

__device__ __forceinline__ float3 sah_centroid(float4 lo, float4 hi) {
    return make_float3(0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z));
}

__global__ void k_sah_init(uint32_t n, int* __restrict__ ids, int* __restrict__ task_of, int first_task) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    ids[i] = (int)i;
    task_of[i] = first_task;
}

__global__ void k_sah_root(uint32_t n, const Bounds* __restrict__ bounds, SahTask* __restrict__ tasks,
                           SahTask* __restrict__ mid, SahSmall* __restrict__ small, SahCounters* __restrict__ ctr) {
    ctr->nodes = 1u;
    ctr->large = 0u;
    ctr->level = n > kSahMidMax ? 1u : 0u;
    ctr->overflow = 0u;
    ctr->mid = n > kSahSeqMax && n <= kSahMidMax ? 1u : 0u;
    if (n > kSahSeqMax) {
        SahTask t;
        t.first = 0u;
        t.count = n;
        t.node = 0;
        t.axis = -1;
        for (int a = 0; a < 3; ++a) {
            t.clo[a] = bounds->lo[a];
            t.chi[a] = bounds->hi[a];
        }
        t.split_bin = 0u;
        t.left_count = 0u;
        t.child_task[0] = t.child_task[1] = -1;
        if (n > kSahMidMax) tasks[0] = t;
        else mid[0] = t;
        ctr->small = 0u;
    } else {
        small[0] = SahSmall{0u, n, 0};
        ctr->small = 1u;
    }
}

__global__ void k_sah_bins_reset(uint32_t words, uint32_t* __restrict__ bins) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= words) return;
    const uint32_t w = i % kSahBinWords;
    // min fields start at the largest ordered value, max fields and counts at 0
    bins[i] = (w < 3 || (w >= 6 && w < 9)) ? 0xffffffffu : 0u;
}

// A warp's triangles into shared bins, `set` the lane's node among those in
// s_bins (< 0: the lane has none). The order is the Morton code's, so
// neighbours fall into the same bins and their atomics would queue up: a run
// that shares its first lane's bin is reduced across the warp and added once.
__device__ __forceinline__ void sah_bins_add(uint32_t* s_bins, int set, float4 lo, float4 hi, float3 c,
                                             const int bin[3]) {
    constexpr uint32_t kFull = 0xffffffffu, kMinGroup = 6u;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t vlo[6] = {float_to_ordered(lo.x), float_to_ordered(lo.y), float_to_ordered(lo.z),
                             float_to_ordered(c.x), float_to_ordered(c.y), float_to_ordered(c.z)};
    const uint32_t vhi[6] = {float_to_ordered(hi.x), float_to_ordered(hi.y), float_to_ordered(hi.z),
                             vlo[3], vlo[4], vlo[5]};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const uint32_t key = set < 0 ? 0xffffffffu : (uint32_t)((set * 3 + a) * kSahBins + bin[a]);
        uint32_t todo = __ballot_sync(kFull, set >= 0);
        for (int g = 0; g < 2 && todo != 0u; ++g) {
            const uint32_t leader = (uint32_t)__ffs(todo) - 1u;
            const uint32_t shared_key = __shfl_sync(kFull, key, leader);
            const uint32_t same = __ballot_sync(kFull, key == shared_key);
            if ((uint32_t)__popc(same) < kMinGroup) break;
            const bool in = key == shared_key;
            uint32_t rlo[6], rhi[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                rlo[k] = __reduce_min_sync(kFull, in ? vlo[k] : 0xffffffffu);
                rhi[k] = __reduce_max_sync(kFull, in ? vhi[k] : 0u);
            }
            if (lane == leader) {
                uint32_t* d = s_bins + shared_key * kSahBinWords;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    atomicMin(d + k, rlo[k]);
                    atomicMax(d + 3 + k, rhi[k]);
                    atomicMin(d + 6 + k, rlo[3 + k]);
                    atomicMax(d + 9 + k, rhi[3 + k]);
                }
                atomicAdd(d + 12, (uint32_t)__popc(same));
            }
            todo &= ~same;
        }
        if ((todo >> lane) & 1u) {
            uint32_t* d = s_bins + key * kSahBinWords;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                atomicMin(d + k, vlo[k]);
                atomicMax(d + 3 + k, vhi[k]);
                atomicMin(d + 6 + k, vlo[3 + k]);
                atomicMax(d + 9 + k, vhi[3 + k]);
            }
            atomicAdd(d + 12, 1u);
        }
    }
}

constexpr int kSahBinPerThread = 2;

// Bins of every triangle in a large node. A block covers kThreads x
// kSahBinPerThread consecutive positions; a large node has more than that, so
// at most two of them meet there, each with its bins in shared memory.
// What bounds it is the shared atomics, which queue on the bins that neighbours
// share. A level of 200k triangles: 16 us; 52 us with every lane's atomics apart
// and one node a block in shared memory.
__global__ void __launch_bounds__(kThreads) k_sah_bin(uint32_t n, const int* __restrict__ ids,
                                                      const int* __restrict__ task_of,
                                                      const SahTask* __restrict__ tasks,
                                                      const float4* __restrict__ leaf_lo,
                                                      const float4* __restrict__ leaf_hi, uint32_t* __restrict__ bins,
                                                      const SahCounters* __restrict__ ctr) {
    static_assert(kThreads * kSahBinPerThread <= kSahMidMax, "two large nodes a block at most");
    __shared__ uint32_t s_bins[2 * kSahTaskWords];
    __shared__ uint32_t s_first[2];
    if (ctr->overflow != 0u) return;  // a level of this batch failed: its lists are not complete
    const uint32_t base = blockIdx.x * (uint32_t)(kThreads * kSahBinPerThread);
    if (threadIdx.x < 2) s_first[threadIdx.x] = 0xffffffffu;
    for (int i = threadIdx.x; i < 2 * kSahTaskWords; i += kThreads) {
        const int w = i % kSahBinWords;
        s_bins[i] = (w < 3 || (w >= 6 && w < 9)) ? 0xffffffffu : 0u;
    }
    __syncthreads();
    int t[kSahBinPerThread];
#pragma unroll
    for (int k = 0; k < kSahBinPerThread; ++k) {
        const uint32_t p = base + (uint32_t)k * kThreads + threadIdx.x;
        t[k] = p < n ? task_of[p] : -1;
        const unsigned live = __ballot_sync(0xffffffffu, t[k] >= 0);
        if (live != 0u && (threadIdx.x & 31u) == (uint32_t)__ffs(live) - 1u) atomicMin(&s_first[0], p);
    }
    __syncthreads();
    if (s_first[0] == 0xffffffffu) return;
    const int first_task = task_of[s_first[0]];
#pragma unroll
    for (int k = 0; k < kSahBinPerThread; ++k) {
        const uint32_t p = base + (uint32_t)k * kThreads + threadIdx.x;
        const unsigned other = __ballot_sync(0xffffffffu, t[k] >= 0 && t[k] != first_task);
        if (other != 0u && (threadIdx.x & 31u) == (uint32_t)__ffs(other) - 1u) atomicMin(&s_first[1], p);
    }
    __syncthreads();
    const int second_task = s_first[1] == 0xffffffffu ? -1 : task_of[s_first[1]];
#pragma unroll
    for (int k = 0; k < kSahBinPerThread; ++k) {
        const uint32_t p = base + (uint32_t)k * kThreads + threadIdx.x;
        const int set = t[k] < 0 ? -1 : t[k] == first_task ? 0 : t[k] == second_task ? 1 : -1;
        float4 lo = make_float4(0.0f, 0.0f, 0.0f, 0.0f), hi = lo;
        float3 c = make_float3(0.0f, 0.0f, 0.0f);
        int bin[3] = {0, 0, 0};
        if (set >= 0) {
            const int prim = ids[p];
            lo = leaf_lo[prim];
            hi = leaf_hi[prim];
            c = sah_centroid(lo, hi);
            const SahTask& task = tasks[t[k]];
            const float cc[3] = {c.x, c.y, c.z};
#pragma unroll
            for (int a = 0; a < 3; ++a)
                bin[a] = sah_bin(cc[a], ordered_to_float(task.clo[a]), ordered_to_float(task.chi[a]));
        }
        sah_bins_add(s_bins, set, lo, hi, c, bin);
    }
    __syncthreads();
    for (int set = 0; set < 2; ++set) {
        const int task = set ? second_task : first_task;
        if (task < 0) break;
        uint32_t* g = bins + (size_t)task * kSahTaskWords;
        for (int i = threadIdx.x; i < kSahTaskWords; i += kThreads) {
            const int w = i % kSahBinWords;
            const uint32_t v = s_bins[set * kSahTaskWords + i];
            if (w < 3 || (w >= 6 && w < 9)) {
                if (v != 0xffffffffu) atomicMin(g + i, v);
            } else if (v != 0u) {
                if (w == 12) atomicAdd(g + i, v);
                else atomicMax(g + i, v);
            }
        }
    }
}

// The split of a node from its bins, by a warp, lane b holding bin b of each
// axis: left and right sweeps as warp scans of the bins' ordered-int boxes and
// counts; the first minimum over axes 0..2, then bins 0..30.
struct SahSplit {
    int axis;  // -1: halve the range
    uint32_t bin, left;
    uint32_t cb[2][6];  // children's centroid bounds
};

static_assert(kSahBins == 32, "one bin per lane");
__device__ __forceinline__ SahSplit sah_best_split(const uint32_t* tb, uint32_t count, const uint32_t clo[3],
                                                   const uint32_t chi[3]) {
    constexpr uint32_t kFull = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u;
    SahSplit out;
    float best_cost = INFINITY;
    int best_axis = -1, best_bin = 0;
    for (int a = 0; a < 3; ++a) {
        const float ext = ordered_to_float(chi[a]) - ordered_to_float(clo[a]);
        if (!(ext > 0.0f)) continue;  // uniform across the warp
        const uint32_t* w = tb + (a * kSahBins + lane) * kSahBinWords;
        // empty bins hold the identities (min fields all ones, max fields 0)
        uint32_t pl[3] = {w[0], w[1], w[2]}, ph[3] = {w[3], w[4], w[5]}, pn = w[12];
        uint32_t sl[3] = {w[0], w[1], w[2]}, sh[3] = {w[3], w[4], w[5]}, sn = w[12];
        for (uint32_t d = 1; d < 32u; d <<= 1) {
            uint32_t ul[3], uh[3], dl[3], dh[3];
            for (int k = 0; k < 3; ++k) {
                ul[k] = __shfl_up_sync(kFull, pl[k], d);
                uh[k] = __shfl_up_sync(kFull, ph[k], d);
                dl[k] = __shfl_down_sync(kFull, sl[k], d);
                dh[k] = __shfl_down_sync(kFull, sh[k], d);
            }
            const uint32_t un = __shfl_up_sync(kFull, pn, d), dn = __shfl_down_sync(kFull, sn, d);
            if (lane >= d) {
                for (int k = 0; k < 3; ++k) {
                    pl[k] = min(pl[k], ul[k]);
                    ph[k] = max(ph[k], uh[k]);
                }
                pn += un;
            }
            if (lane + d < 32u) {
                for (int k = 0; k < 3; ++k) {
                    sl[k] = min(sl[k], dl[k]);
                    sh[k] = max(sh[k], dh[k]);
                }
                sn += dn;
            }
        }
        // split after bin `lane`: left = bins 0..lane (prefix), right = bins lane+1..31
        uint32_t rl[3], rh[3];
        for (int k = 0; k < 3; ++k) {
            rl[k] = __shfl_down_sync(kFull, sl[k], 1);
            rh[k] = __shfl_down_sync(kFull, sh[k], 1);
        }
        const uint32_t rn = __shfl_down_sync(kFull, sn, 1);
        float cost = INFINITY;
        if (lane < 31u && pn != 0u && rn != 0u) {
            const float la = sah_half_area(ordered_to_float(pl[0]), ordered_to_float(pl[1]), ordered_to_float(pl[2]),
                                           ordered_to_float(ph[0]), ordered_to_float(ph[1]), ordered_to_float(ph[2]));
            const float ra = sah_half_area(ordered_to_float(rl[0]), ordered_to_float(rl[1]), ordered_to_float(rl[2]),
                                           ordered_to_float(rh[0]), ordered_to_float(rh[1]), ordered_to_float(rh[2]));
            cost = la * (float)pn + ra * (float)rn;
        }
        float m = cost;
        for (int d = 16; d > 0; d >>= 1) m = fminf(m, __shfl_xor_sync(kFull, m, d));
        if (m < best_cost) {  // strictly cheaper than the earlier axes' best
            best_cost = m;
            best_axis = a;
            best_bin = __ffs(__ballot_sync(kFull, cost == m)) - 1;  // the first bin reaching it
        }
    }
    uint32_t left = count / 2u;
    if (best_axis >= 0) {
        const uint32_t* w = tb + (best_axis * kSahBins + lane) * kSahBinWords;
        const bool in_left = (int)lane <= best_bin;
        left = __reduce_add_sync(kFull, in_left ? w[12] : 0u);
        for (int k = 0; k < 3; ++k) {
            out.cb[0][k] = __reduce_min_sync(kFull, in_left ? w[6 + k] : 0xffffffffu);
            out.cb[0][3 + k] = __reduce_max_sync(kFull, in_left ? w[9 + k] : 0u);
            out.cb[1][k] = __reduce_min_sync(kFull, in_left ? 0xffffffffu : w[6 + k]);
            out.cb[1][3 + k] = __reduce_max_sync(kFull, in_left ? 0u : w[9 + k]);
        }
    } else {
        for (int s = 0; s < 2; ++s)
            for (int k = 0; k < 3; ++k) {
                out.cb[s][k] = clo[k];
                out.cb[s][3 + k] = chi[k];
            }
    }
    out.axis = best_axis;
    out.bin = (uint32_t)best_bin;
    out.left = left;
    return out;
}

// A node's box: the union of its axis-0 bins.
__device__ __forceinline__ void sah_store_box(const uint32_t* tb, int node, float4* node_lo, float4* node_hi) {
    constexpr uint32_t kFull = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t* w = tb + lane * kSahBinWords;
    uint32_t box[6];
    for (int k = 0; k < 3; ++k) {
        box[k] = __reduce_min_sync(kFull, w[k]);
        box[3 + k] = __reduce_max_sync(kFull, w[3 + k]);
    }
    if (lane == 0) {
        node_lo[node] = make_float4(ordered_to_float(box[0]), ordered_to_float(box[1]), ordered_to_float(box[2]), 0.f);
        node_hi[node] = make_float4(ordered_to_float(box[3]), ordered_to_float(box[4]), ordered_to_float(box[5]), 0.f);
    }
}

__device__ __forceinline__ SahTask sah_task(uint32_t first, uint32_t count, int node, const uint32_t cb[6]) {
    SahTask c;
    c.first = first;
    c.count = count;
    c.node = node;
    c.axis = -1;
    for (int k = 0; k < 3; ++k) {
        c.clo[k] = cb[k];
        c.chi[k] = cb[3 + k];
    }
    c.split_bin = 0u;
    c.left_count = 0u;
    c.child_task[0] = c.child_task[1] = -1;
    return c;
}

// One warp per large node: its box, the best split, and the children, which
// lane 0 allocates: interior ids, next-level, mid or small tasks.
__global__ void __launch_bounds__(128) k_sah_split(const uint32_t* __restrict__ count, SahTask* __restrict__ tasks,
                            const uint32_t* __restrict__ bins, SahTask* __restrict__ next, SahTask* __restrict__ mid,
                            SahSmall* __restrict__ small, SahCounters* __restrict__ ctr, SahLimits lim,
                            int2* __restrict__ children, int* __restrict__ node_parent, float4* __restrict__ node_lo,
                            float4* __restrict__ node_hi) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (t >= *count || t >= lim.large || ctr->overflow != 0u) return;  // the whole warp leaves together
    SahTask task = tasks[t];
    const uint32_t* tb = bins + (size_t)t * kSahTaskWords;
    sah_store_box(tb, task.node, node_lo, node_hi);
    const SahSplit split = sah_best_split(tb, task.count, task.clo, task.chi);
    const uint32_t left = split.left;
    if (lane != 0u) return;
    task.axis = split.axis;
    task.split_bin = split.bin;
    task.left_count = left;
    const uint32_t counts[2] = {left, task.count - left};
    int refs[2] = {0, 0};
    for (int s = 0; s < 2; ++s) {
        task.child_task[s] = -1;
        if (counts[s] == 1u) continue;  // a leaf: the scatter writes it
        const int id = (int)atomicAdd(&ctr->nodes, 1u);
        if ((uint32_t)id >= lim.nodes) {
            atomicOr(&ctr->overflow, 1u);
            continue;
        }
        refs[s] = id;
        node_parent[id] = task.node;
        const uint32_t first = task.first + (s ? left : 0u);
        if (counts[s] > kSahMidMax) {
            const uint32_t ti = atomicAdd(&ctr->large, 1u);
            if (ti >= lim.large) {
                atomicOr(&ctr->overflow, 2u);
                continue;
            }
            next[ti] = sah_task(first, counts[s], id, split.cb[s]);
            task.child_task[s] = (int)ti;
        } else if (counts[s] > kSahSeqMax) {
            const uint32_t mi = atomicAdd(&ctr->mid, 1u);
            if (mi >= lim.mid) {
                atomicOr(&ctr->overflow, 32u);
                continue;
            }
            mid[mi] = sah_task(first, counts[s], id, split.cb[s]);
        } else {
            const uint32_t si = atomicAdd(&ctr->small, 1u);
            if (si >= lim.small) {
                atomicOr(&ctr->overflow, 4u);
                continue;
            }
            small[si] = SahSmall{first, counts[s], id};
        }
    }
    if (counts[0] != 1u) children[task.node].x = refs[0];
    if (counts[1] != 1u) children[task.node].y = refs[1];
    tasks[t] = task;
}

__device__ __forceinline__ bool sah_goes_left(const SahTask& task, uint32_t p, const int* ids, const float4* leaf_lo,
                                              const float4* leaf_hi) {
    if (task.axis < 0) return p - task.first < task.left_count;
    const int prim = ids[p];
    const float3 c = sah_centroid(leaf_lo[prim], leaf_hi[prim]);
    const float cc = task.axis == 0 ? c.x : task.axis == 1 ? c.y : c.z;
    const int b = sah_bin(cc, ordered_to_float(task.clo[task.axis]), ordered_to_float(task.chi[task.axis]));
    return (uint32_t)b <= task.split_bin;
}

__global__ void k_sah_flags(uint32_t n, const int* __restrict__ ids, const int* __restrict__ task_of,
                            const SahTask* __restrict__ tasks, const float4* __restrict__ leaf_lo,
                            const float4* __restrict__ leaf_hi, uint32_t* __restrict__ flags,
                            const SahCounters* __restrict__ ctr) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p > n || ctr->overflow != 0u) return;
    uint32_t f = 0u;
    if (p < n) {
        const int t = task_of[p];
        if (t >= 0) f = sah_goes_left(tasks[t], p, ids, leaf_lo, leaf_hi) ? 1u : 0u;
    }
    flags[p] = f;
}

// Stable partition of every large node's range (rank = left flags before the
// position, from an exclusive scan), and the leaves of its children.
__global__ void k_sah_scatter(uint32_t n, const int* __restrict__ ids, const int* __restrict__ task_of,
                              const SahTask* __restrict__ tasks, const uint32_t* __restrict__ flags,
                              const uint32_t* __restrict__ rank, int* __restrict__ ids_out,
                              int* __restrict__ task_of_out, int2* __restrict__ children,
                              int* __restrict__ leaf_parent, SahCounters* __restrict__ ctr) {
    __shared__ bool s_failed;  // an earlier level of the batch: its ids are not complete
    if (threadIdx.x == 0) s_failed = ctr->overflow != 0u;
    __syncthreads();
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n || s_failed) return;
    const int t = task_of[p];
    const int prim = ids[p];
    if (t < 0) {
        ids_out[p] = prim;
        task_of_out[p] = -1;
        return;
    }
    const SahTask& task = tasks[t];
    const uint32_t r = rank[p] - rank[task.first];
    const bool left = flags[p] != 0u;
    // a left rank past the left count (or a right rank past the right count)
    // means the flags and the bins disagree: stop before writing
    if (left ? r >= task.left_count : (p - task.first - r) >= task.count - task.left_count) {
        atomicOr(&ctr->overflow, 8u);
        return;
    }
    const uint32_t q = left ? task.first + r : task.first + task.left_count + (p - task.first - r);
    ids_out[q] = prim;
    const int s = left ? 0 : 1;
    task_of_out[q] = task.child_task[s];
    const uint32_t cn = left ? task.left_count : task.count - task.left_count;
    if (cn == 1u) {
        if (s == 0) children[task.node].x = ~prim;
        else children[task.node].y = ~prim;
        leaf_parent[prim] = task.node;
    }
}

// A block builds a mid node down to small ones: its triangles' order lies in
// shared memory, a stack holds the nodes still to split, and each is binned,
// split by the first warp and partitioned stably, as the large ones are.
// What bounds it is the chain of nodes a block walks, six barriers each. With it
// the 200k-triangle build has 10 levels over the whole GPU instead of 16, each
// six launches and a readback: rebuild 2.85 -> 2.07 ms, this kernel 0.17 ms
// (with k_sah_bin's gain).
struct MidScratch {
    uint32_t bins[kSahTaskWords];
    int ids[kSahMidMax];
    SahTask stack[kSahMidMax / (kSahSeqMax + 1u) + 1u];  // disjoint ranges of more than kSahSeqMax
    SahTask task;
    uint32_t chunk_left[kSahMidMax / 32u];
    int depth;
};

__global__ void __launch_bounds__(kThreads) k_sah_mid(const SahTask* __restrict__ mid, int* __restrict__ ids,
                                                      const float4* __restrict__ leaf_lo,
                                                      const float4* __restrict__ leaf_hi, SahSmall* __restrict__ small,
                                                      SahCounters* __restrict__ ctr, SahLimits lim,
                                                      int2* __restrict__ children, int* __restrict__ node_parent,
                                                      int* __restrict__ leaf_parent, float4* __restrict__ node_lo,
                                                      float4* __restrict__ node_hi) {
    constexpr uint32_t kFull = 0xffffffffu;
    constexpr int kPer = (int)kSahMidMax / kThreads;
    constexpr uint32_t kWarps = kThreads / 32;
    static_assert(kPer * (int)kWarps == 32, "one chunk of 32 positions per lane");
    __shared__ MidScratch m;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t base = mid[blockIdx.x].first, total = mid[blockIdx.x].count;
    if (total > kSahMidMax) {
        if (threadIdx.x == 0) atomicOr(&ctr->overflow, 32u);
        return;  // the whole block
    }
    for (uint32_t r = threadIdx.x; r < total; r += kThreads) m.ids[r] = ids[base + r];
    if (threadIdx.x == 0) {
        m.stack[0] = mid[blockIdx.x];
        m.depth = 1;
    }
    for (;;) {
        __syncthreads();
        const int depth = m.depth;
        if (depth == 0) break;
        const uint32_t first = m.stack[depth - 1].first - base, cnt = m.stack[depth - 1].count;
        const int node = m.stack[depth - 1].node;
        float clo[3], chi[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            clo[a] = ordered_to_float(m.stack[depth - 1].clo[a]);
            chi[a] = ordered_to_float(m.stack[depth - 1].chi[a]);
        }
        for (int i = threadIdx.x; i < kSahTaskWords; i += kThreads) {
            const int w = i % kSahBinWords;
            m.bins[i] = (w < 3 || (w >= 6 && w < 9)) ? 0xffffffffu : 0u;
        }
        __syncthreads();
        int prim[kPer];
        uint32_t bins[kPer];  // axis a in byte a
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const uint32_t r = (uint32_t)k * kThreads + threadIdx.x;
            prim[k] = 0;
            bins[k] = 0u;
            if ((uint32_t)k * kThreads + 32u * warp >= cnt) continue;  // the whole warp
            float4 lo = make_float4(0.0f, 0.0f, 0.0f, 0.0f), hi = lo;
            float3 c = make_float3(0.0f, 0.0f, 0.0f);
            int bin[3] = {0, 0, 0};
            if (r < cnt) {
                prim[k] = m.ids[first + r];
                lo = leaf_lo[prim[k]];
                hi = leaf_hi[prim[k]];
                c = sah_centroid(lo, hi);
                const float cc[3] = {c.x, c.y, c.z};
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    bin[a] = sah_bin(cc[a], clo[a], chi[a]);
                    bins[k] |= (uint32_t)bin[a] << (8 * a);
                }
            }
            sah_bins_add(m.bins, r < cnt ? 0 : -1, lo, hi, c, bin);
        }
        __syncthreads();
        if (warp == 0u) {
            SahTask task = m.stack[depth - 1];
            sah_store_box(m.bins, node, node_lo, node_hi);
            const SahSplit split = sah_best_split(m.bins, cnt, task.clo, task.chi);
            if (lane == 0u) {
                task.axis = split.axis;
                task.split_bin = split.bin;
                task.left_count = split.left;
                const uint32_t counts[2] = {split.left, cnt - split.left};
                int d = depth - 1;
                for (int s = 0; s < 2; ++s) {
                    if (counts[s] == 1u) continue;  // a leaf: the partition writes it
                    const int id = (int)atomicAdd(&ctr->nodes, 1u);
                    if ((uint32_t)id >= lim.nodes) {
                        atomicOr(&ctr->overflow, 1u);
                        continue;
                    }
                    node_parent[id] = node;
                    if (s == 0) children[node].x = id;
                    else children[node].y = id;
                    const uint32_t f = task.first + (s ? split.left : 0u);
                    if (counts[s] > kSahSeqMax) {
                        m.stack[d++] = sah_task(f, counts[s], id, split.cb[s]);
                    } else {
                        const uint32_t si = atomicAdd(&ctr->small, 1u);
                        if (si >= lim.small) {
                            atomicOr(&ctr->overflow, 4u);
                            continue;
                        }
                        small[si] = SahSmall{f, counts[s], id};
                    }
                }
                m.depth = d;
                m.task = task;
            }
        }
        __syncthreads();
        const int axis = m.task.axis;
        const uint32_t split_bin = m.task.split_bin, left = m.task.left_count;
        uint32_t to_left[kPer];
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const uint32_t r = (uint32_t)k * kThreads + threadIdx.x;
            const bool goes = axis < 0 ? r < left : ((bins[k] >> (8 * axis)) & 0xffu) <= split_bin;
            to_left[k] = __ballot_sync(kFull, r < cnt && goes);
            if (lane == 0u) m.chunk_left[(uint32_t)k * kWarps + warp] = (uint32_t)__popc(to_left[k]);
        }
        __syncthreads();
        // left ones before each chunk of 32 positions
        const uint32_t mine = m.chunk_left[lane];
        uint32_t before = mine;
        for (uint32_t d = 1u; d < 32u; d <<= 1) {
            const uint32_t up = __shfl_up_sync(kFull, before, d);
            if (lane >= d) before += up;
        }
        const uint32_t all = __shfl_sync(kFull, before, 31);
        before -= mine;
        if (all != left) {  // the flags and the bins disagree: stop before writing
            if (threadIdx.x == 0) atomicOr(&ctr->overflow, 8u);
            break;  // the whole block
        }
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const uint32_t r = (uint32_t)k * kThreads + threadIdx.x;
            const uint32_t start = __shfl_sync(kFull, before, (uint32_t)k * kWarps + warp);
            if (r >= cnt) continue;
            const uint32_t rank = start + (uint32_t)__popc(to_left[k] & ((1u << lane) - 1u));
            const bool goes = ((to_left[k] >> lane) & 1u) != 0u;
            m.ids[first + (goes ? rank : left + (r - rank))] = prim[k];
            if ((goes ? left : cnt - left) == 1u) {
                if (goes) children[node].x = ~prim[k];
                else children[node].y = ~prim[k];
                leaf_parent[prim[k]] = node;
            }
        }
    }
    for (uint32_t r = threadIdx.x; r < total; r += kThreads) ids[base + r] = m.ids[r];
}

// One warp builds the whole subtree of a small node, with the same split rule.
// The node's boxes lie in shared memory; a node of the subtree is a range of
// their order, lane r (and r + 32) holding its r-th triangle. The best split
// needs no bins: splits between the same two triangles cost the same, and the
// first of them lies after a triangle's own bin, so each lane prices the
// splits after its triangles' bins on the three axes in one pass over the
// range (two shared loads a triangle, broadcast). What bounds it is the chain
// of small nodes a warp walks. One thread a subtree, with its bins in local
// memory, took 2.23 ms of the 200k-triangle build on 38 blocks (6 % of the
// warps); this form takes 0.26 ms (rebuild 4.83 -> 2.90 ms).
constexpr int kSmallWarps = 4;

struct SmallScratch {
    float4 lo[kSahSeqMax], hi[kSahSeqMax];  // box; w: the centroid's x and y
    float cz[kSahSeqMax];
    int prim[kSahSeqMax];
    uint32_t order[kSahSeqMax];
    uint32_t bins[kSahSeqMax];  // by position in the node's range: axis a in byte a
    uint32_t first[kSahSeqMax], count[kSahSeqMax];
    int node[kSahSeqMax];
};

__global__ void __launch_bounds__(32 * kSmallWarps) k_sah_small(
    const uint32_t* __restrict__ count, const SahSmall* __restrict__ small, const int* __restrict__ ids,
    const float4* __restrict__ leaf_lo, const float4* __restrict__ leaf_hi, SahCounters* __restrict__ ctr,
    SahLimits lim, int2* __restrict__ children, int* __restrict__ node_parent, int* __restrict__ leaf_parent,
    float4* __restrict__ node_lo, float4* __restrict__ node_hi) {
    constexpr uint32_t kFull = 0xffffffffu;
    __shared__ SmallScratch scratch[kSmallWarps];
    SmallScratch& m = scratch[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t i = blockIdx.x * kSmallWarps + (threadIdx.x >> 5);
    if (i >= *count || i >= lim.small) return;  // the whole warp leaves together
    const SahSmall root = small[i];
    if (root.count < 2u || root.count > kSahSeqMax) {
        if (lane == 0u) atomicOr(&ctr->overflow, 16u);
        return;
    }
    int next_id = 0;
    if (lane == 0u && root.count > 2u) next_id = (int)atomicAdd(&ctr->nodes, root.count - 2u);
    next_id = __shfl_sync(kFull, next_id, 0);
    if (root.count > 2u && (uint32_t)next_id + (root.count - 2u) > lim.nodes) {
        if (lane == 0u) atomicOr(&ctr->overflow, 1u);
        return;
    }
    for (uint32_t r = lane; r < root.count; r += 32u) {
        const int prim = ids[root.first + r];
        const float4 lo = leaf_lo[prim], hi = leaf_hi[prim];
        const float3 c = sah_centroid(lo, hi);
        // a NaN bound leaves its side of the box open, as fminf / fmaxf do
        m.lo[r] = make_float4(fminf(INFINITY, lo.x), fminf(INFINITY, lo.y), fminf(INFINITY, lo.z), c.x);
        m.hi[r] = make_float4(fmaxf(-INFINITY, hi.x), fmaxf(-INFINITY, hi.y), fmaxf(-INFINITY, hi.z), c.y);
        m.cz[r] = c.z;
        m.prim[r] = prim;
        m.order[r] = r;
    }
    if (lane == 0u) {
        m.first[0] = 0u;
        m.count[0] = root.count;
        m.node[0] = root.node;
    }
    __syncwarp();
    for (int sp = 1; sp > 0;) {
        --sp;
        const uint32_t first = m.first[sp], cnt = m.count[sp];
        const int node = m.node[sp];
        // the lane's triangles, the node's box and its centroid bounds
        uint32_t tri[2];
        float c[2][3];
        float v[12];  // box lo, hi, centroid lo, hi; max fields negated
#pragma unroll
        for (int k = 0; k < 12; ++k) v[k] = INFINITY;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t r = lane + 32u * h;
            tri[h] = 0u;
            c[h][0] = c[h][1] = c[h][2] = 0.0f;
            if (r < cnt) {
                const uint32_t t = m.order[first + r];
                const float4 lo = m.lo[t], hi = m.hi[t];
                tri[h] = t;
                c[h][0] = lo.w;
                c[h][1] = hi.w;
                c[h][2] = m.cz[t];
                v[0] = fminf(v[0], lo.x); v[1] = fminf(v[1], lo.y); v[2] = fminf(v[2], lo.z);
                v[3] = fminf(v[3], -hi.x); v[4] = fminf(v[4], -hi.y); v[5] = fminf(v[5], -hi.z);
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    v[6 + a] = fminf(v[6 + a], c[h][a]);
                    v[9 + a] = fminf(v[9 + a], -c[h][a]);
                }
            }
        }
        for (uint32_t d = 1u; d < 32u && d < cnt; d <<= 1)
#pragma unroll
            for (int k = 0; k < 12; ++k) v[k] = fminf(v[k], __shfl_xor_sync(kFull, v[k], d));
        if (lane == 0u) {
            node_lo[node] = make_float4(v[0], v[1], v[2], 0.0f);
            node_hi[node] = make_float4(-v[3], -v[4], -v[5], 0.0f);
        }
        bool open[3];  // axes whose centroids differ
        uint32_t bins[2] = {0u, 0u};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float cl = __shfl_sync(kFull, v[6 + a], 0), ch = -__shfl_sync(kFull, v[9 + a], 0);
            open[a] = ch - cl > 0.0f;
#pragma unroll
            for (int h = 0; h < 2; ++h) bins[h] |= (uint32_t)sah_bin(c[h][a], cl, ch) << (8 * a);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (lane + 32u * h < cnt) m.bins[lane + 32u * h] = bins[h];
        __syncwarp();
        // the cheapest split: (cost, axis, bin) in that order
        float best_cost = INFINITY;
        uint32_t best_key = 0xffffffffu;  // axis << 8 | bin
        for (int h = 0; h < 2; ++h) {
            if (32u * h >= cnt) break;
            if (lane + 32u * h < cnt) {
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    if (!open[a]) continue;
                    const uint32_t mine = (bins[h] >> (8 * a)) & 0xffu;
                    float ll[3] = {INFINITY, INFINITY, INFINITY}, lh[3] = {-INFINITY, -INFINITY, -INFINITY};
                    float rl[3] = {INFINITY, INFINITY, INFINITY}, rh[3] = {-INFINITY, -INFINITY, -INFINITY};
                    uint32_t ln = 0u;
                    for (uint32_t k = 0; k < cnt; ++k) {
                        const uint32_t t = m.order[first + k];
                        const float4 lo = m.lo[t], hi = m.hi[t];
                        if (((m.bins[k] >> (8 * a)) & 0xffu) <= mine) {
                            ll[0] = fminf(ll[0], lo.x); ll[1] = fminf(ll[1], lo.y); ll[2] = fminf(ll[2], lo.z);
                            lh[0] = fmaxf(lh[0], hi.x); lh[1] = fmaxf(lh[1], hi.y); lh[2] = fmaxf(lh[2], hi.z);
                            ++ln;
                        } else {
                            rl[0] = fminf(rl[0], lo.x); rl[1] = fminf(rl[1], lo.y); rl[2] = fminf(rl[2], lo.z);
                            rh[0] = fmaxf(rh[0], hi.x); rh[1] = fmaxf(rh[1], hi.y); rh[2] = fmaxf(rh[2], hi.z);
                        }
                    }
                    if (ln == cnt) continue;
                    const float cost = sah_half_area(ll[0], ll[1], ll[2], lh[0], lh[1], lh[2]) * (float)ln +
                                       sah_half_area(rl[0], rl[1], rl[2], rh[0], rh[1], rh[2]) * (float)(cnt - ln);
                    const uint32_t key = ((uint32_t)a << 8) | mine;
                    if (cost < best_cost || (cost == best_cost && key < best_key)) {
                        best_cost = cost;
                        best_key = key;
                    }
                }
            }
        }
        float least = best_cost;
        for (int d = 16; d > 0; d >>= 1) least = fminf(least, __shfl_xor_sync(kFull, least, d));
        // no lane has a split below infinity: halve the range
        const uint32_t key = __reduce_min_sync(kFull, best_cost == least && least < INFINITY ? best_key : 0xffffffffu);
        // stable partition of the range
        uint32_t to_left[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t r = lane + 32u * h;
            const bool goes = key != 0xffffffffu ? ((bins[h] >> (8u * (key >> 8))) & 0xffu) <= (key & 0xffu)
                                                 : r < cnt / 2u;
            to_left[h] = __ballot_sync(kFull, r < cnt && goes);
        }
        __syncwarp();  // the order is read above and written below
        const uint32_t left = (uint32_t)(__popc(to_left[0]) + __popc(to_left[1]));
        const uint32_t below = (1u << lane) - 1u;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t r = lane + 32u * h;
            if (r >= cnt) continue;
            const uint32_t rank = (uint32_t)__popc(to_left[h] & below) + (h ? (uint32_t)__popc(to_left[0]) : 0u);
            m.order[first + (((to_left[h] >> lane) & 1u) ? rank : left + (r - rank))] = tri[h];
        }
        __syncwarp();
        // the children, by lane 0: leaves, or ranges to build next
        const uint32_t counts[2] = {left, cnt - left};
        int refs[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t f = first + (h ? left : 0u);
            if (counts[h] == 1u) {
                const int prim = m.prim[m.order[f]];
                refs[h] = ~prim;
                if (lane == 0u) leaf_parent[prim] = node;
            } else {
                const int id = next_id++;
                refs[h] = id;
                if (lane == 0u) {
                    node_parent[id] = node;
                    m.first[sp] = f;
                    m.count[sp] = counts[h];
                    m.node[sp] = id;
                }
                ++sp;
            }
        }
        if (lane == 0u) children[node] = make_int2(refs[0], refs[1]);
        __syncwarp();
    }
}

template <class T> T* dmalloc(size_t count, cudaStream_t s, cudaError_t* err) {
    void* p = nullptr;
    cudaError_t e = nan_host::scratch_alloc(&p, std::max<size_t>(count, 1) * sizeof(T), s);
    if (e != cudaSuccess && *err == cudaSuccess) *err = e;
    return static_cast<T*>(p);
}

uint32_t blocks(uint64_t n) { return (uint32_t)((n + kThreads - 1) / kThreads); }

}  // namespace

namespace nan_host {

void forget_scene(NanContext* ctx) {
    ctx->wide_count = 0;
    ctx->wide_built = false;
    ctx->has_scene = false;
    ctx->tri_count = ctx->node_count = ctx->leaf_count = ctx->max_depth = 0;
}

void free_scene(NanContext* ctx) {
    if (!ctx->caller_owned_bvh) {
        cudaFree(ctx->nodes);
        cudaFree(ctx->tris);
        cudaFree(ctx->tri_refs);
    }
    cudaFree(ctx->wnodes);
    cudaFree(ctx->wtris);
    ctx->wnodes = nullptr;
    ctx->wtris = nullptr;
    ctx->caller_owned_bvh = false;
    ctx->nodes = nullptr;
    ctx->tris = nullptr;
    ctx->tri_refs = nullptr;
    ctx->bvh_capacity = ctx->wide_capacity = 0;
    ctx->device_bytes = 0;
    forget_scene(ctx);
}


int finish_binary(NanContext* ctx, uint32_t n, const float4* tris_sorted, const float4* leaf_lo,
                  const float4* leaf_hi, int2* children, int* node_parent, int* leaf_parent, float4* node_lo,
                  float4* node_hi, uint32_t* arrivals, uint32_t* depth, double* sah, const Bounds* bounds,
                  const int* root_dev, cudaStream_t s);

// Binned-SAH hierarchy over the leaves (kernels k_sah_*): large nodes level by
// level, one host readback of the next level's node count per kSahBatch
// levels, then the mid nodes and the small nodes in one launch each; the root
// is interior node 0.
int build_binned(NanContext* ctx, uint32_t n, const float4* tris_sorted, const float4* leaf_lo,
                 const float4* leaf_hi, int2* children, int* node_parent, int* leaf_parent, float4* node_lo,
                 float4* node_hi, uint32_t* arrivals, uint32_t* depth, double* sah, const Bounds* bounds,
                 cudaStream_t s) {
    cudaError_t err = cudaSuccess;
    const uint32_t max_large = n / (kSahMidMax + 1u) + 1u, max_mid = n / (kSahSeqMax + 1u) + 1u;
    const SahLimits lim{max_large, n / 2u + 1u, n - 1u, max_mid};
    int* ids_a = dmalloc<int>(n, s, &err);
    int* ids_b = dmalloc<int>(n, s, &err);
    int* task_a = dmalloc<int>(n, s, &err);
    int* task_b = dmalloc<int>(n, s, &err);
    uint32_t* flags = dmalloc<uint32_t>(n + 1, s, &err);
    uint32_t* rank = dmalloc<uint32_t>(n + 1, s, &err);
    SahTask* level_a = dmalloc<SahTask>(max_large, s, &err);
    SahTask* level_b = dmalloc<SahTask>(max_large, s, &err);
    SahTask* mid = dmalloc<SahTask>(max_mid, s, &err);
    SahSmall* small = dmalloc<SahSmall>(n / 2u + 1u, s, &err);
    uint32_t* bins = dmalloc<uint32_t>((size_t)max_large * kSahTaskWords, s, &err);
    SahCounters* ctr = dmalloc<SahCounters>(1, s, &err);
    int* root_dev = dmalloc<int>(1, s, &err);
    size_t scan_bytes = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, flags, rank, n + 1, s);
    void* scan_tmp = dmalloc<uint8_t>(scan_bytes, s, &err);
    auto release = [&] {
        for (void* p : {(void*)ids_a, (void*)ids_b, (void*)task_a, (void*)task_b, (void*)flags, (void*)rank,
                        (void*)level_a, (void*)level_b, (void*)mid, (void*)small, (void*)bins, (void*)ctr, (void*)root_dev,
                        scan_tmp})
            if (p) cudaFreeAsync(p, s);
    };
    // every exit releases the scratch
    auto fail = [&](cudaError_t e, const char* what) {
        release();
        return cuda_fail(e, what);
    };
    auto limit = [&](const char* what) {
        release();
        set_error(what);
        return NAN_ERR_LIMIT;
    };
    if (err != cudaSuccess) return fail(err, "binned SAH scratch allocation");
    cudaMemsetAsync(root_dev, 0, sizeof(int), s);
    cudaMemsetAsync(node_parent, 0xff, (n - 1u) * sizeof(int), s);  // the root's parent stays -1
    k_sah_init<<<blocks(n), kThreads, 0, s>>>(n, ids_a, task_a, n > kSahMidMax ? 0 : -1);
    k_sah_root<<<1, 1, 0, s>>>(n, bounds, level_a, mid, small, ctr);
    ctx->launches += 2;
    uint32_t large = n > kSahMidMax ? 1u : 0u;
    int levels = 0;
    const uint32_t bin_grid = (uint32_t)((n + kThreads * kSahBinPerThread - 1) / (kThreads * kSahBinPerThread));
    // Levels run in batches of kSahBatch without the host: a level has at most
    // twice the nodes of the one before, and its kernels read the count itself.
    // 200k triangles, 10 levels: rebuild 1.82 -> 1.70 ms; in batches of three, two
    // of whose levels then find nothing to do, 1.74.
    while (large > 0u) {
        uint32_t bound = large;
        for (int k = 0; k < kSahBatch; ++k) {
            if (++levels > kSahMaxLevels) return limit("binned SAH build did not terminate");
            const uint32_t words = bound * (uint32_t)kSahTaskWords;
            k_sah_bins_reset<<<blocks(words), kThreads, 0, s>>>(words, bins);
            k_sah_bin<<<bin_grid, kThreads, 0, s>>>(n, ids_a, task_a, level_a, leaf_lo, leaf_hi, bins, ctr);
            k_sah_split<<<(bound * 32u + 127u) / 128u, 128, 0, s>>>(&ctr->level, level_a, bins, level_b, mid, small,
                                                                    ctr, lim, children, node_parent, node_lo, node_hi);
            k_sah_flags<<<blocks(n + 1), kThreads, 0, s>>>(n, ids_a, task_a, level_a, leaf_lo, leaf_hi, flags, ctr);
            cub::DeviceScan::ExclusiveSum(scan_tmp, scan_bytes, flags, rank, n + 1, s);
            k_sah_scatter<<<blocks(n), kThreads, 0, s>>>(n, ids_a, task_a, level_a, flags, rank, ids_b, task_b,
                                                         children, leaf_parent, ctr);
            ctx->launches += 6;
            // the next level's count becomes the current one
            cudaMemcpyAsync(&ctr->level, &ctr->large, sizeof(uint32_t), cudaMemcpyDeviceToDevice, s);
            err = cudaMemsetAsync(&ctr->large, 0, sizeof(uint32_t), s);
            if (err != cudaSuccess) return fail(err, "binned SAH level");
            std::swap(ids_a, ids_b);
            std::swap(task_a, task_b);
            std::swap(level_a, level_b);
            bound = std::min(2u * bound, max_large);
        }
        SahCounters lc{};
        err = cudaMemcpyAsync(&lc, ctr, sizeof(SahCounters), cudaMemcpyDeviceToHost, s);
        if (err == cudaSuccess) err = cudaStreamSynchronize(s);
        if (err != cudaSuccess) return fail(err, "binned SAH level");
        large = lc.level;
        if (lc.overflow != 0u || large > max_large) return limit("binned SAH build exceeded a bound of its node lists");
    }
    SahCounters c{};
    err = cudaMemcpyAsync(&c, ctr, sizeof(SahCounters), cudaMemcpyDeviceToHost, s);
    if (err == cudaSuccess) err = cudaStreamSynchronize(s);
    if (err != cudaSuccess) return fail(err, "binned SAH counters");
    if (c.overflow != 0u || c.mid > max_mid) return limit("binned SAH build exceeded a bound of its node lists");
    if (c.mid > 0u) {
        k_sah_mid<<<c.mid, kThreads, 0, s>>>(mid, ids_a, leaf_lo, leaf_hi, small, ctr, lim, children, node_parent,
                                             leaf_parent, node_lo, node_hi);
        ctx->launches++;
        err = cudaMemcpyAsync(&c, ctr, sizeof(SahCounters), cudaMemcpyDeviceToHost, s);
        if (err == cudaSuccess) err = cudaStreamSynchronize(s);
        if (err != cudaSuccess) return fail(err, "binned SAH mid nodes");
        if (c.overflow != 0u) return limit("binned SAH build exceeded a bound of its node lists");
    }
    if (c.small > 0u) {
        k_sah_small<<<(c.small + kSmallWarps - 1u) / kSmallWarps, 32 * kSmallWarps, 0, s>>>(&ctr->small, small, ids_a, leaf_lo, leaf_hi, ctr, lim,
                                                             children, node_parent, leaf_parent, node_lo, node_hi);
        ctx->launches++;
    }
    err = cudaMemcpyAsync(&c, ctr, sizeof(SahCounters), cudaMemcpyDeviceToHost, s);
    if (err == cudaSuccess) err = cudaStreamSynchronize(s);
    if (err != cudaSuccess) return fail(err, "binned SAH small nodes");
    if (c.overflow != 0u || c.nodes != n - 1u) return limit("binned SAH build made the wrong number of interior nodes");
    const int rc = finish_binary(ctx, n, tris_sorted, leaf_lo, leaf_hi, children, node_parent, leaf_parent, node_lo,
                                 node_hi, arrivals, depth, sah, bounds, root_dev, s);
    release();
    return rc;
}

// PLOC hierarchy over the Morton-sorted leaves, SAH leaf collapse, and a
// depth-first emission of nodes and triangles (see the kernels above).
int build_ploc(NanContext* ctx, uint32_t n, const float4* tris_sorted, const float4* leaf_lo, const float4* leaf_hi,
               int2* children, int* node_parent, int* leaf_parent, float4* node_lo, float4* node_hi,
               uint32_t* arrivals, uint32_t* depth, double* sah, const Bounds* bounds, cudaStream_t s) {
    cudaError_t err = cudaSuccess;
    const uint32_t interior = n - 1;
    int* idx_a = dmalloc<int>(n, s, &err);
    int* idx_b = dmalloc<int>(n, s, &err);
    float4* lo_a = dmalloc<float4>(n, s, &err);
    float4* hi_a = dmalloc<float4>(n, s, &err);
    float4* lo_b = dmalloc<float4>(n, s, &err);
    float4* hi_b = dmalloc<float4>(n, s, &err);
    int* nn = dmalloc<int>(n, s, &err);
    uint32_t* valid = dmalloc<uint32_t>(n + 1, s, &err);
    uint32_t* pos = dmalloc<uint32_t>(n + 1, s, &err);
    // [0] interior nodes made; [1], [2] live clusters (double-buffered)
    uint32_t* counter = dmalloc<uint32_t>(3, s, &err);
    size_t scan_bytes = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, valid, pos, n + 1, s);
    void* scan_tmp = dmalloc<uint8_t>(scan_bytes, s, &err);
    if (err != cudaSuccess) return cuda_fail(err, "PLOC scratch allocation");
    cudaMemsetAsync(node_parent, 0xff, interior * sizeof(int), s);
    {
        const uint32_t init[3] = {0u, n, n};
        cudaMemcpyAsync(counter, init, sizeof(init), cudaMemcpyHostToDevice, s);
    }
    cudaMemsetAsync(valid, 0, (n + 1) * sizeof(uint32_t), s);
    k_ploc_init<<<blocks(n), kThreads, 0, s>>>(n, idx_a);
    cudaMemcpyAsync(lo_a, leaf_lo, n * sizeof(float4), cudaMemcpyDeviceToDevice, s);
    cudaMemcpyAsync(hi_a, leaf_hi, n * sizeof(float4), cudaMemcpyDeviceToDevice, s);
    ctx->launches++;
    // Iterations run in batches of kPlocBatch without the host: each kernel
    // reads the live count (counter[1]); the host reads it back once per
    // batch to size the next batch's grids and to check progress.
    uint32_t c = n;
    int iterations = 0;
    while (c > 1) {
        if (iterations > 4096) {
            set_error("PLOC did not converge");
            return NAN_ERR_LIMIT;
        }
        const uint32_t grid = (c + kPlocBlock - 1) / kPlocBlock;
        for (int k = 0; k < kPlocBatch; ++k, ++iterations) {
            uint32_t* live = counter + 1 + (iterations & 1);
            uint32_t* next_live = counter + 1 + ((iterations + 1) & 1);
            k_ploc_nn<<<grid, kPlocBlock, 0, s>>>(live, lo_a, hi_a, nn);
            k_ploc_merge<<<blocks(c + 1), kThreads, 0, s>>>(live, (int)c, nn, idx_a, lo_a, hi_a, idx_b, lo_b, hi_b,
                                                            valid, children, node_parent, leaf_parent, node_lo,
                                                            node_hi, counter);
            cub::DeviceScan::ExclusiveSum(scan_tmp, scan_bytes, valid, pos, c + 1, s);
            k_ploc_compact<<<blocks(c), kThreads, 0, s>>>(live, next_live, valid, pos, idx_b, lo_b, hi_b, idx_a,
                                                          lo_a, hi_a);
            ctx->launches += 4;
        }
        uint32_t next = 0;
        // kPlocBatch is even, so after a batch the live count is in slot 1 + 0
        err = cudaMemcpyAsync(&next, counter + 1 + (iterations & 1), sizeof(uint32_t), cudaMemcpyDeviceToHost, s);
        if (err == cudaSuccess) err = cudaStreamSynchronize(s);
        if (err != cudaSuccess) return cuda_fail(err, "PLOC iteration");
        if (next >= c) {
            set_error("PLOC made no progress");
            return NAN_ERR_LIMIT;
        }
        c = next;
    }
    const int rc = finish_binary(ctx, n, tris_sorted, leaf_lo, leaf_hi, children, node_parent, leaf_parent, node_lo,
                                 node_hi, arrivals, depth, sah, bounds, idx_a, s);
    for (void* p : {(void*)idx_a, (void*)idx_b, (void*)lo_a, (void*)hi_a, (void*)lo_b, (void*)hi_b, (void*)nn,
                    (void*)valid, (void*)pos, (void*)counter, scan_tmp})
        cudaFreeAsync(p, s);
    return rc;
}

// SAH leaf collapse, depth-first emission of nodes and triangles, and the
// compressed 8-wide conversion of a binary hierarchy over the n leaves
// (children / parents / interior boxes; root_dev[0] is the root's index).
int finish_binary(NanContext* ctx, uint32_t n, const float4* tris_sorted, const float4* leaf_lo,
                  const float4* leaf_hi, int2* children, int* node_parent, int* leaf_parent, float4* node_lo,
                  float4* node_hi, uint32_t* arrivals, uint32_t* depth, double* sah, const Bounds* bounds,
                  const int* root_dev, cudaStream_t s) {
    cudaError_t err = cudaSuccess;
    const uint32_t interior = n - 1;
    SubtreeInfo* info = dmalloc<SubtreeInfo>(interior, s, &err);
    int* dfs = dmalloc<int>(interior, s, &err);
    uint32_t* tri_off = dmalloc<uint32_t>(interior, s, &err);
    uint32_t* tri_pos = dmalloc<uint32_t>(n, s, &err);
    if (err != cudaSuccess) return cuda_fail(err, "BVH collapse scratch allocation");
    int root = 0;
    err = cudaMemcpyAsync(&root, root_dev, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (err == cudaSuccess) err = cudaStreamSynchronize(s);
    if (err != cudaSuccess) return cuda_fail(err, "BVH root readback");
    cudaMemsetAsync(arrivals, 0, interior * sizeof(uint32_t), s);
    k_subtree<<<blocks(n), kThreads, 0, s>>>(n, children, node_parent, leaf_parent, leaf_lo, leaf_hi, node_lo, node_hi,
                                            info, arrivals);
    k_dfs_nodes<<<blocks(interior), kThreads, 0, s>>>(interior, children, node_parent, info, dfs, tri_off);
    k_dfs_leaves<<<blocks(n), kThreads, 0, s>>>(n, children, node_parent, leaf_parent, info, tri_pos);
    k_scatter_tris<<<blocks(n), kThreads, 0, s>>>(n, tri_pos, tris_sorted, ctx->tris);
    err = cudaGetLastError();
    if (err != cudaSuccess) return cuda_fail(err, "BVH collapse");

    // compressed 8-wide BVH from the collapsed binary tree, level by level
    if (ctx->wide_capacity < n) {
        cudaFree(ctx->wnodes);
        cudaFree(ctx->wtris);
        ctx->wnodes = nullptr;
        ctx->wtris = nullptr;
        ctx->wide_capacity = 0;
        if (cudaMalloc(&ctx->wnodes, (size_t)n * 5 * sizeof(uint4)) != cudaSuccess ||
            cudaMalloc(&ctx->wtris, (size_t)n * 3 * sizeof(float4)) != cudaSuccess) {
            set_error("out of device memory for the wide BVH");
            return NAN_ERR_OUT_OF_MEMORY;
        }
        ctx->device_bytes += (uint64_t)n * (5 * sizeof(uint4) + 3 * sizeof(float4));
        ctx->wide_capacity = n;
    }
    WideItem* items_a = dmalloc<WideItem>(interior + 1, s, &err);
    WideItem* items_b = dmalloc<WideItem>(interior + 1, s, &err);
    // [0] wide nodes, [1] wide triangles, [2 + l] items of level l
    uint32_t* wcount = dmalloc<uint32_t>(2 + kWideMaxLevels + 1, s, &err);
    if (err != cudaSuccess) return cuda_fail(err, "wide BVH scratch allocation");
    {
        // the root item: the binary root; levels run in batches of
        // kWideBatch without the host, each grid bounded by 8x the last
        k_wide_root<<<1, 1, 0, s>>>(root_dev, items_a);
        cudaMemsetAsync(wcount, 0, (2 + kWideMaxLevels + 1) * sizeof(uint32_t), s);
        const uint32_t init[3] = {1u, 0u, 1u};
        cudaMemcpyAsync(wcount, init, sizeof(init), cudaMemcpyHostToDevice, s);
        uint64_t bound = 1;
        int level = 0;
        for (;;) {
            for (int k = 0; k < kWideBatch; ++k, ++level) {
                if (level >= kWideMaxLevels) {
                    set_error("wide BVH conversion did not terminate");
                    return NAN_ERR_LIMIT;
                }
                const WideItem* in = (level & 1) ? items_b : items_a;
                WideItem* out = (level & 1) ? items_a : items_b;
                k_wide_level<<<blocks(bound * kWideLanes), kThreads, 0, s>>>(in, wcount + 2 + level, out, wcount + 3 + level,
                                                                wcount, children, node_lo, node_hi, leaf_lo, leaf_hi,
                                                                info, tri_off, tri_pos, ctx->tris, bounds,
                                                                ctx->wnodes, ctx->wtris);
                ctx->launches++;
                bound = std::min<uint64_t>(bound * 8u, (uint64_t)interior + 1u);
            }
            uint32_t pending = 0;
            err = cudaMemcpyAsync(&pending, wcount + 2 + level, sizeof(uint32_t), cudaMemcpyDeviceToHost, s);
            if (err == cudaSuccess) err = cudaMemcpyAsync(&ctx->wide_count, wcount, sizeof(uint32_t),
                                                          cudaMemcpyDeviceToHost, s);
            if (err == cudaSuccess) err = cudaStreamSynchronize(s);
            if (err != cudaSuccess) return cuda_fail(err, "wide BVH level");
            if (pending == 0u) break;
        }
        ctx->wide_built = true;
    }
    cudaFreeAsync(items_a, s);
    cudaFreeAsync(items_b, s);
    cudaFreeAsync(wcount, s);
    k_emit_dfs<<<blocks(interior), kThreads, 0, s>>>(interior, children, node_lo, node_hi, leaf_lo, leaf_hi, bounds,
                                                     info, dfs, tri_off, tri_pos, root, ctx->nodes, sah);
    k_depth<<<blocks(n), kThreads, 0, s>>>(n, node_parent, leaf_parent, depth);
    ctx->launches += 6;
    SubtreeInfo root_info;
    uint32_t max_depth = 0;
    double sah_host = 0.0;
    err = cudaMemcpyAsync(&root_info, info + root, sizeof(SubtreeInfo), cudaMemcpyDeviceToHost, s);
    if (err == cudaSuccess) err = cudaMemcpyAsync(&max_depth, depth, sizeof(uint32_t), cudaMemcpyDeviceToHost, s);
    if (err == cudaSuccess) err = cudaMemcpyAsync(&sah_host, sah, sizeof(double), cudaMemcpyDeviceToHost, s);
    if (err == cudaSuccess) err = cudaStreamSynchronize(s);
    if (err != cudaSuccess) return cuda_fail(err, "BVH emit");
    for (void* p : {(void*)info, (void*)dfs, (void*)tri_off, (void*)tri_pos}) cudaFreeAsync(p, s);
    if (root_info.collapsed) {  // the whole scene is one leaf
        ctx->root = ~(int)(n - 1u);
        ctx->node_count = 0;
        ctx->sah_cost = (double)n;
    } else {
        ctx->root = 0;
        ctx->node_count = root_info.interior;
        ctx->sah_cost = sah_host;
    }
    ctx->leaf_count = n;
    ctx->max_depth = max_depth;
    return NAN_OK;
}

int build_scene(NanContext* ctx, const NanSceneDesc* sd, cudaStream_t s) {
    cudaError_t err = cudaSuccess;
    if (ctx->caller_owned_bvh) free_scene(ctx);  // never reuse caller memory
    else forget_scene(ctx);
    ctx->scene = *sd;
    const uint32_t I = sd->instance_count;

    cudaEvent_t ev0, ev1;
    cudaEventCreate(&ev0);
    cudaEventCreate(&ev1);
    cudaEventRecord(ev0, s);

    // 1. flat offsets
    uint32_t* counts = dmalloc<uint32_t>(I + 1, s, &err);
    uint32_t* offsets = dmalloc<uint32_t>(I + 1, s, &err);
    if (err != cudaSuccess) return cuda_fail(err, "scene build allocation");
    k_instance_counts<<<blocks(I + 1), kThreads, 0, s>>>(reinterpret_cast<const uint4*>(sd->instance_descs),
                                                         reinterpret_cast<const uint4*>(sd->mesh_descs), I, counts);
    ctx->launches++;
    size_t scan_bytes = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, counts, offsets, I + 1, s);
    void* scan_tmp = dmalloc<uint8_t>(scan_bytes, s, &err);
    cub::DeviceScan::ExclusiveSum(scan_tmp, scan_bytes, counts, offsets, I + 1, s);
    ctx->launches++;
    uint32_t total = 0;
    err = cudaMemcpyAsync(&total, offsets + I, sizeof(uint32_t), cudaMemcpyDeviceToHost, s);
    if (err == cudaSuccess) err = cudaStreamSynchronize(s);
    if (err != cudaSuccess) return cuda_fail(err, "scene build (triangle count)");
    cudaFreeAsync(scan_tmp, s);
    cudaFreeAsync(counts, s);
    if (total > (1u << 30)) {
        cudaFreeAsync(offsets, s);
        set_error("scene has more than 2^30 triangles");
        return NAN_ERR_INVALID_ARGUMENT;
    }
    const uint32_t n = total;
    ctx->tri_count = n;

    // Persistent storage, kept from an earlier build when it is large enough.
    const uint32_t interior = n > 1 ? n - 1 : 0;
    const uint32_t cap = std::max<uint32_t>(n, 1);
    if (ctx->bvh_capacity < cap) {
        cudaFree(ctx->tris);
        cudaFree(ctx->tri_refs);
        cudaFree(ctx->nodes);
        ctx->tris = nullptr;
        ctx->tri_refs = nullptr;
        ctx->nodes = nullptr;
        ctx->bvh_capacity = 0;
        if (cudaMalloc(&ctx->tris, (size_t)cap * 3 * sizeof(float4)) != cudaSuccess ||
            cudaMalloc(&ctx->tri_refs, (size_t)cap * sizeof(uint2)) != cudaSuccess ||
            cudaMalloc(&ctx->nodes, (size_t)cap * 4 * sizeof(float4)) != cudaSuccess) {
            cudaFreeAsync(offsets, s);
            free_scene(ctx);
            set_error("out of device memory for the BVH");
            return NAN_ERR_OUT_OF_MEMORY;
        }
        ctx->bvh_capacity = cap;
    }
    ctx->device_bytes = (uint64_t)ctx->bvh_capacity * (3 * sizeof(float4) + sizeof(uint2) + 4 * sizeof(float4)) +
                        (uint64_t)ctx->wide_capacity * (5 * sizeof(uint4) + 3 * sizeof(float4));

    if (n == 0) {
        cudaFreeAsync(offsets, s);
        ctx->has_scene = true;
        ctx->root = 0;
        cudaEventDestroy(ev0);
        cudaEventDestroy(ev1);
        return NAN_OK;
    }

    // Scratch.
    float4* tris_flat = dmalloc<float4>(3ull * n, s, &err);
    float4* lo_flat = dmalloc<float4>(n, s, &err);
    float4* hi_flat = dmalloc<float4>(n, s, &err);
    Bounds* bounds = dmalloc<Bounds>(1, s, &err);
    uint64_t* keys = dmalloc<uint64_t>(n, s, &err);
    uint64_t* keys_sorted = dmalloc<uint64_t>(n, s, &err);
    uint32_t* vals = dmalloc<uint32_t>(n, s, &err);
    uint32_t* order = dmalloc<uint32_t>(n, s, &err);
    float4* leaf_lo = dmalloc<float4>(n, s, &err);
    float4* leaf_hi = dmalloc<float4>(n, s, &err);
    int2* children = dmalloc<int2>(std::max<uint32_t>(interior, 1), s, &err);
    int* node_parent = dmalloc<int>(std::max<uint32_t>(interior, 1), s, &err);
    int* leaf_parent = dmalloc<int>(n, s, &err);
    float4* node_lo = dmalloc<float4>(std::max<uint32_t>(interior, 1), s, &err);
    float4* node_hi = dmalloc<float4>(std::max<uint32_t>(interior, 1), s, &err);
    uint32_t* arrivals = dmalloc<uint32_t>(std::max<uint32_t>(interior, 1), s, &err);
    uint32_t* depth = dmalloc<uint32_t>(1, s, &err);
    double* sah = dmalloc<double>(1, s, &err);
    if (err != cudaSuccess) return cuda_fail(err, "scene build scratch allocation");

    Bounds init;
    for (int a = 0; a < 3; ++a) {
        init.lo[a] = 0xffffffffu;
        init.hi[a] = 0u;
    }
    init.max_abs = 0u;
    cudaMemcpyAsync(bounds, &init, sizeof(Bounds), cudaMemcpyHostToDevice, s);
    cudaMemsetAsync(arrivals, 0, std::max<uint32_t>(interior, 1) * sizeof(uint32_t), s);
    cudaMemsetAsync(depth, 0, sizeof(uint32_t), s);
    cudaMemsetAsync(sah, 0, sizeof(double), s);

    // 2-3. flatten + bounds
    k_flatten<<<blocks(n), kThreads, 0, s>>>(*sd, offsets, n, tris_flat, ctx->tri_refs, lo_flat, hi_flat, bounds);
    // 4. Morton codes + sort
    k_morton<<<blocks(n), kThreads, 0, s>>>(lo_flat, hi_flat, n, bounds, keys, vals);
    size_t sort_bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, keys, keys_sorted, vals, order, (int)n, 0, 63, s);
    void* sort_tmp = dmalloc<uint8_t>(sort_bytes, s, &err);
    if (err != cudaSuccess) return cuda_fail(err, "scene build sort allocation");
    cub::DeviceRadixSort::SortPairs(sort_tmp, sort_bytes, keys, keys_sorted, vals, order, (int)n, 0, 63, s);
    // NanTuning.bvh_builder: 0 binned SAH, 1 LBVH, 2 PLOC
    const bool use_sah = ctx->tuning.bvh_builder == 0 && n > 1;
    const bool use_ploc = ctx->tuning.bvh_builder == 2 && n > 1;
    float4* tris_sorted = (use_sah || use_ploc) ? dmalloc<float4>(3ull * n, s, &err) : ctx->tris;
    if (err != cudaSuccess) return cuda_fail(err, "scene build scratch allocation");
    k_gather_leaves<<<blocks(n), kThreads, 0, s>>>(order, n, tris_flat, lo_flat, hi_flat, tris_sorted, leaf_lo, leaf_hi);
    ctx->launches += 4;
    if (n == 1) {
        ctx->root = ~0;
        ctx->node_count = 0;
        ctx->leaf_count = 1;
        ctx->max_depth = 1;
        ctx->sah_cost = 1.0;
    } else if (use_sah || use_ploc) {
        int rc = use_sah ? build_binned(ctx, n, tris_sorted, leaf_lo, leaf_hi, children, node_parent, leaf_parent,
                                        node_lo, node_hi, arrivals, depth, sah, bounds, s)
                         : build_ploc(ctx, n, tris_sorted, leaf_lo, leaf_hi, children, node_parent, leaf_parent,
                                      node_lo, node_hi, arrivals, depth, sah, bounds, s);
        cudaFreeAsync(tris_sorted, s);
        if (rc != NAN_OK) return rc;
    } else {
        // 5-7. hierarchy, refit, depth, emit
        k_hierarchy<<<blocks(interior), kThreads, 0, s>>>(keys_sorted, (int)n, children, node_parent, leaf_parent);
        k_refit<<<blocks(n), kThreads, 0, s>>>(n, children, node_parent, leaf_parent, leaf_lo, leaf_hi, node_lo,
                                               node_hi, arrivals);
        k_depth<<<blocks(n), kThreads, 0, s>>>(n, node_parent, leaf_parent, depth);
        k_emit<<<blocks(interior), kThreads, 0, s>>>(interior, children, node_lo, node_hi, leaf_lo, leaf_hi, bounds,
                                                     ctx->nodes, sah);
        ctx->launches += 4;
        ctx->root = 0;
        ctx->node_count = interior;
        ctx->leaf_count = n;
        uint32_t max_depth = 0;
        double sah_host = 0.0;
        err = cudaMemcpyAsync(&max_depth, depth, sizeof(uint32_t), cudaMemcpyDeviceToHost, s);
        if (err == cudaSuccess) err = cudaMemcpyAsync(&sah_host, sah, sizeof(double), cudaMemcpyDeviceToHost, s);
        if (err == cudaSuccess) err = cudaStreamSynchronize(s);
        if (err != cudaSuccess) return cuda_fail(err, "scene build (depth and SAH readback)");
        ctx->max_depth = max_depth;
        ctx->sah_cost = sah_host;
    }
    cudaEventRecord(ev1, s);
    for (void* p : {(void*)offsets, (void*)tris_flat, (void*)lo_flat, (void*)hi_flat, (void*)bounds, (void*)keys,
                    (void*)keys_sorted, (void*)vals, (void*)order, (void*)leaf_lo, (void*)leaf_hi, (void*)children,
                    (void*)node_parent, (void*)leaf_parent, (void*)node_lo, (void*)node_hi, (void*)arrivals,
                    (void*)depth, (void*)sah, sort_tmp})
        cudaFreeAsync(p, s);
    err = cudaStreamSynchronize(s);
    if (err != cudaSuccess) return cuda_fail(err, "scene build");
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, ev0, ev1);
    ctx->build_ms = ms;
    cudaEventDestroy(ev0);
    cudaEventDestroy(ev1);
    if (ctx->max_depth > 96u) {
        set_error("BVH deeper than the traversal stack (96)");
        free_scene(ctx);
        return NAN_ERR_LIMIT;
    }
    ctx->has_scene = true;
    return NAN_OK;
}

namespace {
__global__ void k_world_tris(const float4* __restrict__ tris, uint32_t n, float* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 a = tris[3u * i], b = tris[3u * i + 1], c = tris[3u * i + 2];
    const uint32_t f = __float_as_uint(a.w);
    float* o = out + 9ull * f;
    o[0] = a.x; o[1] = a.y; o[2] = a.z;
    o[3] = b.x; o[4] = b.y; o[5] = b.z;
    o[6] = c.x; o[7] = c.y; o[8] = c.z;
}
}  // namespace

int world_triangles(NanContext* ctx, float* out, cudaStream_t s) {
    if (ctx->tri_count == 0) return NAN_OK;
    k_world_tris<<<blocks(ctx->tri_count), kThreads, 0, s>>>(ctx->tris, ctx->tri_count, out);
    ctx->launches++;
    return cuda_fail(cudaGetLastError(), "world triangles");
}

}  // namespace nan_host

// ---------------------------------------------------------------------------
// nan_scene_build_noalloc: the scene build for callers that cannot allocate
// device memory (code running where cudaMalloc is unavailable or forbidden,
// e.g. inside another framework's memory pool or a real-time loop that must
// never allocate). All scratch lives in the fixed array below; the BVH goes
// into caller-provided buffers.
// ---------------------------------------------------------------------------
namespace {

// Scratch shared by every nan_scene_build_noalloc call on a device. The CUDA
// loader places one copy on each GPU that loads this library, held until the
// process exits. Calls that overlap on the GPU race on it.
constexpr size_t kNoAllocScratchBytes = 64ull << 20;
__device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

// Device address of g_noalloc_scratch per device ordinal. In host code the
// symbol is only a host-side stand-in, so the address comes from
// cudaGetSymbolAddress, taken once per device with that device current. The
// cached address belongs to the device's primary context: after
// cudaDeviceReset it is stale, and the library must not be used for a
// no-alloc build on that device again in this process.
std::mutex g_noalloc_mutex;
void* g_noalloc_address[128] = {};

int noalloc_scratch(int device, unsigned char** out) {
    if (device < 0 || device >= 128) {
        set_error("device ordinal out of range for the no-alloc scratch table");
        return NAN_ERR_INVALID_ARGUMENT;
    }
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (g_noalloc_address[device] == nullptr) {
        void* p = nullptr;
        const cudaError_t err = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (err != cudaSuccess) return cuda_fail(err, "cudaGetSymbolAddress(no-alloc scratch)");
        g_noalloc_address[device] = p;
    }
    *out = static_cast<unsigned char*>(g_noalloc_address[device]);
    return NAN_OK;
}

// Bump carving of the static scratch, 256-byte aligned.
struct Carver {
    unsigned char* base;
    size_t used = 0;
    size_t capacity;
    template <class T> T* take(size_t count) {
        used = (used + 255u) & ~size_t(255u);
        T* p = reinterpret_cast<T*>(base + used);
        used += std::max<size_t>(count, 1) * sizeof(T);
        return p;
    }
    bool fits() const { return used <= capacity; }
};

}  // namespace

extern "C" NAN_B200_API int nan_scene_build_noalloc(NanContext* ctx, const NanSceneDesc* sd, float* out_nodes,
                                                    uint64_t nodes_bytes, float* out_tris, uint64_t tris_bytes,
                                                    uint32_t* out_refs, uint64_t refs_bytes, void* stream) {
    if (!ctx || !sd) {
        set_error("null context or scene description");
        return NAN_ERR_INVALID_ARGUMENT;
    }
    cudaError_t err = cudaSetDevice(ctx->device);
    if (err != cudaSuccess) return cuda_fail(err, "cudaSetDevice");
    if (!ctx->caller_owned_bvh && (ctx->nodes || ctx->tris || ctx->tri_refs)) {
        set_error("context holds a BVH allocated by nan_scene_build; use a context without one");
        return NAN_ERR_INVALID_ARGUMENT;
    }
    // Forget the previous caller-owned BVH without freeing anything.
    auto forget_bvh = [ctx]() {
        ctx->nodes = nullptr;
        ctx->tris = nullptr;
        ctx->tri_refs = nullptr;
        ctx->caller_owned_bvh = false;
        ctx->has_scene = false;
        ctx->tri_count = ctx->node_count = ctx->leaf_count = ctx->max_depth = 0;
        ctx->device_bytes = 0;
    };
    if (sd->instance_count == 0 || !sd->vertices || !sd->indices || !sd->mesh_descs || !sd->instance_descs ||
        !sd->transforms || !sd->inverse_transposes || !sd->materials) {
        set_error("scene needs at least one instance and non-null buffers");
        return NAN_ERR_INVALID_ARGUMENT;
    }
    if (!out_nodes || !out_tris || !out_refs || (reinterpret_cast<uintptr_t>(out_nodes) & 15u) ||
        (reinterpret_cast<uintptr_t>(out_tris) & 15u) || (reinterpret_cast<uintptr_t>(out_refs) & 7u)) {
        set_error("output buffers must be non-null; nodes and tris 16-byte aligned, refs 8-byte aligned");
        return NAN_ERR_INVALID_ARGUMENT;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    unsigned char* scratch = nullptr;
    int rc = noalloc_scratch(ctx->device, &scratch);
    if (rc) return rc;
    const uint32_t I = sd->instance_count;

    // Triangle count (per-instance counts + scan in the scratch).
    Carver head{scratch, 0, kNoAllocScratchBytes};
    uint32_t* counts = head.take<uint32_t>(I + 1);
    uint32_t* offsets = head.take<uint32_t>(I + 1);
    size_t scan_bytes = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, counts, offsets, I + 1, s);
    unsigned char* scan_tmp = head.take<unsigned char>(scan_bytes);
    if (!head.fits()) {
        set_error("too many instances for the no-alloc scratch (64 MiB)");
        return NAN_ERR_LIMIT;
    }
    k_instance_counts<<<blocks(I + 1), kThreads, 0, s>>>(reinterpret_cast<const uint4*>(sd->instance_descs),
                                                         reinterpret_cast<const uint4*>(sd->mesh_descs), I, counts);
    cub::DeviceScan::ExclusiveSum(scan_tmp, scan_bytes, counts, offsets, I + 1, s);
    ctx->launches += 2;
    uint32_t n = 0;
    err = cudaMemcpyAsync(&n, offsets + I, sizeof(uint32_t), cudaMemcpyDeviceToHost, s);
    if (err == cudaSuccess) err = cudaStreamSynchronize(s);
    if (err != cudaSuccess) return cuda_fail(err, "no-alloc scene build (triangle count)");
    if (n == 0) {
        set_error("scene has no triangles");
        return NAN_ERR_INVALID_ARGUMENT;
    }
    const uint32_t interior = n > 1 ? n - 1 : 0;
    if (nodes_bytes < (uint64_t)std::max<uint32_t>(interior, 1) * 64u || tris_bytes < (uint64_t)n * 48u ||
        refs_bytes < (uint64_t)n * 8u) {
        set_error("output buffers too small: need 64*max(T-1,1) node, 48*T triangle and 8*T ref bytes");
        return NAN_ERR_INVALID_ARGUMENT;
    }

    // Carve the rest of the build's scratch after the offsets.
    Carver c = head;
    float4* tris_flat = c.take<float4>(3ull * n);
    float4* lo_flat = c.take<float4>(n);
    float4* hi_flat = c.take<float4>(n);
    Bounds* bounds = c.take<Bounds>(1);
    uint64_t* keys = c.take<uint64_t>(n);
    uint64_t* keys_sorted = c.take<uint64_t>(n);
    uint32_t* vals = c.take<uint32_t>(n);
    uint32_t* order = c.take<uint32_t>(n);
    float4* leaf_lo = c.take<float4>(n);
    float4* leaf_hi = c.take<float4>(n);
    int2* children = c.take<int2>(interior);
    int* node_parent = c.take<int>(interior);
    int* leaf_parent = c.take<int>(n);
    float4* node_lo = c.take<float4>(interior);
    float4* node_hi = c.take<float4>(interior);
    uint32_t* arrivals = c.take<uint32_t>(interior);
    uint32_t* depth = c.take<uint32_t>(1);
    double* sah = c.take<double>(1);
    size_t sort_bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, keys, keys_sorted, vals, order, (int)n, 0, 63, s);
    unsigned char* sort_tmp = c.take<unsigned char>(sort_bytes);
    if (!c.fits()) {
        set_error("scene too large for the no-alloc scratch (64 MiB, about 300k triangles)");
        return NAN_ERR_LIMIT;
    }

    // Previous calls leave their contents behind: clear what must start at zero.
    Bounds init;
    for (int a = 0; a < 3; ++a) {
        init.lo[a] = 0xffffffffu;
        init.hi[a] = 0u;
    }
    init.max_abs = 0u;
    err = cudaMemcpyAsync(bounds, &init, sizeof(Bounds), cudaMemcpyHostToDevice, s);
    if (err == cudaSuccess) err = cudaMemsetAsync(arrivals, 0, std::max<uint32_t>(interior, 1) * sizeof(uint32_t), s);
    if (err == cudaSuccess) err = cudaMemsetAsync(depth, 0, sizeof(uint32_t), s);
    if (err == cudaSuccess) err = cudaMemsetAsync(sah, 0, sizeof(double), s);
    if (err != cudaSuccess) return cuda_fail(err, "no-alloc scene build (scratch clear)");

    forget_bvh();
    ctx->scene = *sd;
    ctx->caller_owned_bvh = true;
    ctx->nodes = reinterpret_cast<float4*>(out_nodes);
    ctx->tris = reinterpret_cast<float4*>(out_tris);
    ctx->tri_refs = reinterpret_cast<uint2*>(out_refs);
    ctx->tri_count = n;
    ctx->device_bytes = 0;

    k_flatten<<<blocks(n), kThreads, 0, s>>>(*sd, offsets, n, tris_flat, ctx->tri_refs, lo_flat, hi_flat, bounds);
    k_morton<<<blocks(n), kThreads, 0, s>>>(lo_flat, hi_flat, n, bounds, keys, vals);
    cub::DeviceRadixSort::SortPairs(sort_tmp, sort_bytes, keys, keys_sorted, vals, order, (int)n, 0, 63, s);
    k_gather_leaves<<<blocks(n), kThreads, 0, s>>>(order, n, tris_flat, lo_flat, hi_flat, ctx->tris, leaf_lo, leaf_hi);
    ctx->launches += 4;
    uint32_t max_depth = 1;
    double sah_host = 1.0;
    if (n == 1) {
        ctx->root = ~0;
        ctx->node_count = 0;
    } else {
        k_hierarchy<<<blocks(interior), kThreads, 0, s>>>(keys_sorted, (int)n, children, node_parent, leaf_parent);
        k_refit<<<blocks(n), kThreads, 0, s>>>(n, children, node_parent, leaf_parent, leaf_lo, leaf_hi, node_lo,
                                               node_hi, arrivals);
        k_depth<<<blocks(n), kThreads, 0, s>>>(n, node_parent, leaf_parent, depth);
        k_emit<<<blocks(interior), kThreads, 0, s>>>(interior, children, node_lo, node_hi, leaf_lo, leaf_hi, bounds,
                                                     ctx->nodes, sah);
        ctx->launches += 4;
        ctx->root = 0;
        ctx->node_count = interior;
        err = cudaMemcpyAsync(&max_depth, depth, sizeof(uint32_t), cudaMemcpyDeviceToHost, s);
        if (err == cudaSuccess) err = cudaMemcpyAsync(&sah_host, sah, sizeof(double), cudaMemcpyDeviceToHost, s);
        if (err != cudaSuccess) {
            forget_bvh();
            return cuda_fail(err, "no-alloc scene build (depth and SAH readback)");
        }
    }
    err = cudaStreamSynchronize(s);
    if (err != cudaSuccess) {
        forget_bvh();
        return cuda_fail(err, "no-alloc scene build");
    }
    ctx->leaf_count = n;
    ctx->max_depth = max_depth;
    ctx->sah_cost = sah_host;
    ctx->build_ms = 0.0;
    if (ctx->max_depth > 96u) {
        forget_bvh();
        set_error("BVH deeper than the traversal stack (96)");
        return NAN_ERR_LIMIT;
    }
    ctx->has_scene = true;
    return NAN_OK;
}
