// nan_wavefront.cu -- wavefront form of the integrators.
//
// A path lives in SoA state arrays between kernels. Each round runs:
//   trace  persistent warps pull rays from two compacted queues: the closest
//          hit of every walking path's ray, and any hit of the shadow rays
//          that the last round's stage queued, adding the contributions of
//          the visible ones;
//   stage  per path: emission, sun NEE shadow ray (queued), next direction;
//          a path that ended one round ago, or left the scene now, is closed
//          (and starts the next sample or side, or retires).
// A path that ends at a surface has its last shadow ray in flight while the
// others trace on, and is closed a round later. Shadow and closest-hit rays
// of neighbouring vertices thus share one launch: two launches and one wait
// for the longest ray per round, where a launch each for extend, shade,
// shadow and finalize took four and two.
// The RNG of a path is the reference's per-thread stream, drawn in the same
// order, and every radiance sum is formed in the same order as the
// reference's loop, so the result equals the one-thread-per-unit kernels bit
// for bit. Compiled with --fmad=false (see nan_math.cuh).
#include <algorithm>
#include <cstring>

#include "nan_internal.h"
#include "nan_scene.cuh"
#include "nan_sinks.cuh"
#include "nan_probe.cuh"

namespace {

using namespace nbd;
using nan_host::cuda_fail;
using nan_host::set_error;

constexpr uint32_t kFlagBack = 1u << 0;
constexpr uint32_t kFlagNoPath = 1u << 2;
constexpr uint32_t kFlagTwoSided = 1u << 3;
constexpr uint32_t kBounceShift = 4;
constexpr uint32_t kBounceMask = 0xffu << kBounceShift;
constexpr uint32_t kSampleShift = 12;

constexpr uint32_t kKindNee = 0u;  // shadow contribution goes to rad
constexpr uint32_t kKindSun = 1u;  // shadow contribution goes to si (screen: the area-light term)

struct WfState {
    uint32_t* unit;   // surface texel / probe index
    uint32_t* rng;
    uint32_t* flags;
    float4* surf;     // b1, b2, instance bits, primitive bits
    float4* ro;       // origin, w = t_min
    float4* rd;       // direction, w = t_max
    float4* thp;
    float4* rad;
    float4* si;
    float4* irr;
    float2* zpdf;     // |z| and pdf of the sample's first direction
    float4* hit;      // flat bits (~0 = miss), t, b1, b2
    float4* pa;       // probes: source instance bits, source primitive bits, source offset, first-hit distance
    uint4* pb;        // probes: self-hit suspects of the sample, of all samples, previous count, radial texel
    uint4* pc;        // probes: 2 per path, per-radial-texel sample counts (16 x u16)
};

// Queues of one chunk of paths. The paths that trace on fill a round's extend
// queue from the front, those that wait to be closed from the back: each path
// in flight is in it at most once.
struct WfQueues {
    uint32_t* ext[2];
    uint32_t* ext_sorted;  // the extend queue regrouped by direction octant (NanTuning ray_order 1)
    float4* shd[2];        // 3 float4 per entry: (o, path bits), (d, kind bits), (c, 0)
    uint32_t* ctl;         // kCtlWords per round: kExt, kExtFetch, kShd, kShdFetch, kClose
    uint32_t* oct;         // 8 paths per octant, 8 placement cursors
    uint32_t cap;          // paths in flight: the length of an extend queue
};

// Words of a round's control block: walking paths, fetch counter of the trace
// (or extend) launch, shadow rays queued by the round's stage, fetch counter
// of a separate shadow launch, paths to close.
constexpr uint32_t kCtlWords = 8u, kExt = 0u, kExtFetch = 1u, kShd = 2u, kShdFetch = 3u, kClose = 4u;

constexpr size_t kBytesPerPath = 4 + 4 + 4 + 16 * 9 + 8 + 16 + 16 + 32 + 3 * 4 + 2 * 2 * 48;

// Warp-aggregated append: returns this lane's slot in the queue.
__device__ __forceinline__ uint32_t queue_slot(uint32_t* count, bool want) {
    const unsigned active = __activemask();
    const unsigned mask = __ballot_sync(active, want);
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t base = 0u;
    const int leader = __ffs(mask) - 1;
    if (mask && (int)lane == leader) base = atomicAdd(count, (uint32_t)__popc(mask));
    base = __shfl_sync(active, base, leader < 0 ? __ffs(active) - 1 : leader);
    return base + (uint32_t)__popc(mask & ((1u << lane) - 1u));
}

// Appends of a whole block to up to two queues: counts per warp, one atomic
// per queue and block, then every thread its slot. Every thread of the block
// calls it; two blocks of shared memory taken in turn need no further barrier
// between calls. Appending by warp left the queues a patchwork of part warps
// and made every warp wait for its turn at one address. By block, neighbouring
// paths stay together in the queues (trace launches of the 200k-triangle texel
// iteration 15.2 -> 14.3 ms, all of it 19.65 -> 18.78 ms) and a chunk of 2 M
// screen paths is generated in 31 us (177 us; its queue needs no atomics at
// all). Blocks of 128 threads; 256 take 18.87 ms.
constexpr int kStageThreads = 128;

struct BlockAppend {
    uint32_t n[2][kStageThreads / 32];
    uint32_t base[2];
};

__device__ __forceinline__ uint2 block_slots(BlockAppend& sh, uint32_t* count0, bool want0, uint32_t* count1,
                                             bool want1) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const unsigned m0 = __ballot_sync(0xffffffffu, want0), m1 = __ballot_sync(0xffffffffu, want1);
    if (lane == 0u) {
        sh.n[0][warp] = (uint32_t)__popc(m0);
        sh.n[1][warp] = (uint32_t)__popc(m1);
    }
    __syncthreads();
    if (lane == 0u && warp < 2u) {
        uint32_t sum = 0u;
#pragma unroll
        for (int w = 0; w < kStageThreads / 32; ++w) sum += sh.n[warp][w];
        if (sum) sh.base[warp] = atomicAdd(warp ? count1 : count0, sum);
    }
    __syncthreads();
    uint2 slot = make_uint2(sh.base[0], sh.base[1]);
    for (uint32_t w = 0; w < warp; ++w) {
        slot.x += sh.n[0][w];
        slot.y += sh.n[1][w];
    }
    const unsigned below = (1u << lane) - 1u;
    slot.x += (uint32_t)__popc(m0 & below);
    slot.y += (uint32_t)__popc(m1 & below);
    return slot;
}

// What becomes of a path after a stage: it retires, traces on in the next
// round, or waits there to be closed.
enum PathNext { kRetire = 0, kWalk = 1, kAwaitClose = 2 };

// The block's paths into the queue of the round that (buf, ctl) belong to:
// the walking ones from the front, those to close from the back.
__device__ __forceinline__ void push_paths(BlockAppend& sh, const WfQueues& q, int buf, uint32_t* ctl, uint32_t p,
                                           PathNext next) {
    const uint2 slot = block_slots(sh, ctl + kExt, next == kWalk, ctl + kClose, next == kAwaitClose);
    if (next == kWalk) q.ext[buf][slot.x] = p;
    if (next == kAwaitClose) q.ext[buf][q.cap - 1u - slot.y] = p;
}

// Slots in the shadow queue of the round that ctl belongs to.
__device__ __forceinline__ uint32_t shadow_slots(BlockAppend& sh, uint32_t* ctl, bool want) {
    return block_slots(sh, ctl + kShd, want, nullptr, false).x;
}

// Counters of the generated units (context counters 2 and 3), by block.
__device__ __forceinline__ void count_units(unsigned long long* counters, bool unit, uint32_t paths) {
    __shared__ uint32_t s_paths;
    const int units = __syncthreads_count(unit);
    if (threadIdx.x == 0u) s_paths = 0u;
    __syncthreads();
    const uint32_t sum = __reduce_add_sync(0xffffffffu, unit ? paths : 0u);
    if ((threadIdx.x & 31u) == 0u && sum) atomicAdd(&s_paths, sum);
    __syncthreads();
    if (threadIdx.x == 0u && units) {
        atomicAdd(counters + 2, (unsigned long long)units);
        atomicAdd(counters + 3, (unsigned long long)s_paths);
    }
}

// A shadow ray at its slot; tmax 0: the ray runs to the scene's t_max.
__device__ __forceinline__ void store_shadow(const WfQueues& q, int buf, uint32_t slot, uint32_t p, f3 o, f3 d, f3 c,
                                             uint32_t kind, float tmax = 0.0f) {
    float4* e = q.shd[buf] + 3u * slot;
    e[0] = make_float4(o.x, o.y, o.z, __uint_as_float(p));
    e[1] = make_float4(d.x, d.y, d.z, __uint_as_float(kind));
    e[2] = make_float4(c.x, c.y, c.z, tmax);
}

__device__ __forceinline__ f3 xyz(float4 v) { return mk3(v.x, v.y, v.z); }
__device__ __forceinline__ float4 f4(f3 v, float w) { return make_float4(v.x, v.y, v.z, w); }

// ---------------------------------------------------------------------------
// Generic traversal stages.
// ---------------------------------------------------------------------------
// Extend-queue regrouping by ray direction octant (x < 0 | y < 0 << 1 |
// z < 0 << 2): neighbouring lanes of the traversal then follow rays of one
// octant, in their previous order within it. Two passes over the queue:
// a histogram, then a placement with warp-aggregated cursors.
__device__ __forceinline__ uint32_t dir_octant(float4 d) {
    return (d.x < 0.0f ? 1u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 4u : 0u);
}

__global__ void __launch_bounds__(256) k_wf_octant_count(const uint32_t* __restrict__ queue, const uint32_t* ctl,
                                                         const float4* __restrict__ rd, uint32_t* oct) {
    const uint32_t count = *(volatile const uint32_t*)(ctl + kExt);
    for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < count; idx += gridDim.x * blockDim.x) {
        const uint32_t o = dir_octant(rd[queue[idx]]);
        const unsigned group = __match_any_sync(__activemask(), o);
        if ((threadIdx.x & 31u) == (uint32_t)(__ffs(group) - 1)) atomicAdd(oct + o, (uint32_t)__popc(group));
    }
}

__global__ void __launch_bounds__(256) k_wf_octant_place(const uint32_t* __restrict__ queue, const uint32_t* ctl,
                                                         const float4* __restrict__ rd, uint32_t* oct,
                                                         uint32_t* __restrict__ out) {
    const uint32_t count = *(volatile const uint32_t*)(ctl + kExt);
    uint32_t base[8];
    uint32_t sum = 0u;
    for (int o = 0; o < 8; ++o) {
        base[o] = sum;
        sum += oct[o];
    }
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < count; idx += gridDim.x * blockDim.x) {
        const uint32_t p = queue[idx];
        const uint32_t o = dir_octant(rd[p]);
        const unsigned active = __activemask();
        const unsigned group = __match_any_sync(active, o);
        const int leader = __ffs(group) - 1;
        uint32_t first = 0u;
        if ((int)lane == leader) first = atomicAdd(oct + 8 + o, (uint32_t)__popc(group));
        first = __shfl_sync(active, first, leader);
        out[base[o] + first + (uint32_t)__popc(group & ((1u << lane) - 1u))] = p;
    }
}

// The paths to close of a regrouped queue, at its back as before.
__global__ void __launch_bounds__(256) k_wf_close_copy(const uint32_t* __restrict__ queue, const uint32_t* ctl,
                                                       uint32_t cap, uint32_t* __restrict__ out) {
    const uint32_t count = *(volatile const uint32_t*)(ctl + kClose);
    for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < count; idx += gridDim.x * blockDim.x)
        out[cap - 1u - idx] = queue[cap - 1u - idx];
}

// Scene of a path: one scene for the per-scene passes, the path's probe set
// for the multi-scene batch (set index per path).
struct OneScene {
    SceneView s;
    __device__ __forceinline__ const SceneView& of(uint32_t) const { return s; }
};

struct ManyScenes {
    const BatchSet* sets;
    const uint32_t* set_of;
    __device__ __forceinline__ const SceneView& of(uint32_t p) const { return sets[set_of[p]].s; }
};

// Rays a warp takes from a queue at once: 32, or fewer where the queue would
// leave warps of the grid without any: then the even share. Few rays a warp
// end sooner: a warp runs as long as its longest ray, and its diverging lanes
// take turns (probe baker over 20,480 sites: 9.1 ms with 32 rays a warp, 5.8
// with the even share, extend and shadow in launches of their own). Warps take
// their first rays by their number, without an atomic.
__device__ __forceinline__ uint32_t rays_per_grab(unsigned long long count) {
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    return (uint32_t)min(32ull, max(1ull, (count + warps - 1u) / warps));
}

// Traversal forms. kShared > 0 (binary nodes): the first kShared
// traversal-stack entries of a thread live in a shared-memory column
// (stack_top, of the thread), the rest in local memory. kSpec (binary nodes):
// the speculative while-while walk.
template <int kWidth, int kShared, bool kSpec>
__device__ __forceinline__ HitInfo closest_form(const SceneView& s, int* stack_top, f3 o, f3 d, float tmin,
                                                float tmax) {
    if constexpr (kShared > 0 && kWidth == 2) {
        SplitStack<kShared, 128, kTraversalStack + 2> stk;
        stk.top = stack_top;
        return trace_closest_binary_s<kTraversalStack>(s, stk, o, d, tmin, tmax);
    } else if constexpr (kSpec && kWidth == 2) {
        return trace_closest_binary_spec(s, o, d, tmin, tmax);
    } else {
        return trace_closest_w<kWidth>(s, o, d, tmin, tmax);
    }
}

template <int kWidth, int kShared, bool kSpec>
__device__ __forceinline__ bool any_form(const SceneView& s, int* stack_top, f3 o, f3 d, float tmax) {
    if constexpr (kShared > 0 && kWidth == 2) {
        SplitStack<kShared, 128, kTraversalStack + 2> stk;
        stk.top = stack_top;
        return trace_any_binary_s<kTraversalStack>(s, stk, o, d, 0.0f, tmax);
    } else if constexpr (kSpec && kWidth == 2) {
        return trace_any_binary_spec(s, o, d, 0.0f, tmax);
    } else {
        return trace_any_w<kWidth>(s, o, d, 0.0f, tmax);
    }
}

// The two kinds of rays as a launch each, for stage timing; their launch bounds
// are k_wf_trace's.
template <int kWidth, class Src, int kShared = 0, bool kSpec = false>
__global__ void __launch_bounds__(128, 9) k_wf_extend(Src src, const uint32_t* __restrict__ queue,
                                                   uint32_t* ctl, const float4* __restrict__ ro,
                                                   const float4* __restrict__ rd, float4* __restrict__ hit,
                                                   unsigned long long* counters) {
    const uint32_t count = *(volatile uint32_t*)(ctl + kExt);
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t grab = rays_per_grab(count);
    RayTally tally{0u, 0u};
    __shared__ int stack_top[kShared > 0 ? kShared * 128 : 1];
    const uint32_t warps = gridDim.x * (blockDim.x >> 5), first = warps * grab;
    for (uint32_t base = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * grab; base < count;) {
        const uint32_t idx = base + lane;
        if (lane < grab && idx < count) {
            const uint32_t p = queue[idx];
            const SceneView s = src.of(p);
            const float4 o = ro[p], d = rd[p];
            tally.extend++;
            const HitInfo h =
                closest_form<kWidth, kShared, kSpec>(s, stack_top + threadIdx.x, xyz(o), xyz(d), o.w, d.w);
            hit[p] = make_float4(__uint_as_float(h.valid ? h.flat : 0xffffffffu), h.t, h.b1, h.b2);
        }
        if (first >= count) break;
        if (lane == 0u) base = atomicAdd(ctl + kExtFetch, grab);
        base = first + __shfl_sync(0xffffffffu, base, 0);
    }
    flush_tally(counters, tally, 0u, 0u);
}

template <int kWidth, class Src, int kShared = 0, bool kSpec = false>
__global__ void __launch_bounds__(128, 9) k_wf_shadow(Src src, const float4* __restrict__ queue, uint32_t* ctl,
                                                   float t_max, float4* __restrict__ rad, float4* __restrict__ si,
                                                   unsigned long long* counters) {
    const uint32_t count = *(volatile uint32_t*)(ctl + kShd);
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t grab = rays_per_grab(count);
    RayTally tally{0u, 0u};
    __shared__ int stack_top[kShared > 0 ? kShared * 128 : 1];
    const uint32_t warps = gridDim.x * (blockDim.x >> 5), first = warps * grab;
    for (uint32_t base = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * grab; base < count;) {
        const uint32_t idx = base + lane;
        if (lane < grab && idx < count) {
            const float4 a = queue[3u * idx], b = queue[3u * idx + 1u], c = queue[3u * idx + 2u];
            tally.shadow++;
            const uint32_t p = __float_as_uint(a.w);
            const SceneView s = src.of(p);
            const bool blocked = any_form<kWidth, kShared, kSpec>(s, stack_top + threadIdx.x, xyz(a), xyz(b),
                                                                  c.w > 0.0f ? c.w : t_max);
            if (!blocked) {
                float4* target = (__float_as_uint(b.w) == kKindNee) ? rad : si;
                const float4 v = target[p];
                target[p] = make_float4(v.x + c.x, v.y + c.y, v.z + c.z, v.w);
            }
        }
        if (first >= count) break;
        if (lane == 0u) base = atomicAdd(ctl + kShdFetch, grab);
        base = first + __shfl_sync(0xffffffffu, base, 0);
    }
    flush_tally(counters, tally, 0u, 0u);
}

// The trace launch of a round: the closest hits of the walking paths (ctl) and
// the shadow rays of the round before (ctl_prev). Warps take chunks of up to
// 32 rays of one kind, closest hits first. Against extend, shade, shadow and
// finalize launches in turn: probe baker over 20,480 sites 6.14 -> 4.77 ms,
// 256x256 box frame 267 -> 200 us, 1080p frame over 1M triangles
// 2.71 -> 2.43 ms, 200k-triangle texel iteration 20.0 -> 19.6 ms. The other
// forms and widths that take whole grabs run the same way (8-wide nodes, a
// 640x480 frame over 82k triangles 1.16 -> 0.91 ms).
// 9 resident blocks of 128 per SM (56 registers a thread): the 200k-triangle
// texel iteration takes 18.85 ms, against 19.06 with 8 blocks and 19.87 with 10
// (48 registers, spills), the 16-scene probe batch 14.01, 14.25 and 15.40, the
// 1080p frame 2.25, 2.27 and 2.37, the probe baker 4.81, 4.73 and 4.99.
template <int kWidth, class Src, int kShared = 0, bool kSpec = false>
__global__ void __launch_bounds__(128, 9) k_wf_trace(Src src, const uint32_t* __restrict__ queue, uint32_t* ctl,
                                                     const float4* __restrict__ ro, const float4* __restrict__ rd,
                                                     float4* __restrict__ hit, const float4* __restrict__ shadows,
                                                     const uint32_t* ctl_prev, float t_max, float4* __restrict__ rad,
                                                     float4* __restrict__ si, unsigned long long* counters) {
    const uint32_t rays = *(volatile uint32_t*)(ctl + kExt);
    const uint32_t shadow_rays = *(const volatile uint32_t*)(ctl_prev + kShd);
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t grab = rays_per_grab((unsigned long long)rays + shadow_rays);
    const uint32_t ray_chunks = (rays + grab - 1u) / grab, chunks = ray_chunks + (shadow_rays + grab - 1u) / grab;
    RayTally tally{0u, 0u};
    __shared__ int stack_top[kShared > 0 ? kShared * 128 : 1];
    for (uint32_t c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < chunks;) {
        if (c < ray_chunks) {
            const uint32_t idx = c * grab + lane;
            if (lane < grab && idx < rays) {
                const uint32_t p = queue[idx];
                const SceneView s = src.of(p);
                const float4 o = ro[p], d = rd[p];
                tally.extend++;
                const HitInfo h =
                    closest_form<kWidth, kShared, kSpec>(s, stack_top + threadIdx.x, xyz(o), xyz(d), o.w, d.w);
                hit[p] = make_float4(__uint_as_float(h.valid ? h.flat : 0xffffffffu), h.t, h.b1, h.b2);
            }
        } else {
            const uint32_t idx = (c - ray_chunks) * grab + lane;
            if (lane < grab && idx < shadow_rays) {
                const float4 a = shadows[3u * idx], b = shadows[3u * idx + 1u], e = shadows[3u * idx + 2u];
                tally.shadow++;
                const uint32_t p = __float_as_uint(a.w);
                const SceneView s = src.of(p);
                if (!any_form<kWidth, kShared, kSpec>(s, stack_top + threadIdx.x, xyz(a), xyz(b),
                                                      e.w > 0.0f ? e.w : t_max)) {
                    float4* target = (__float_as_uint(b.w) == kKindNee) ? rad : si;
                    const float4 v = target[p];
                    target[p] = make_float4(v.x + e.x, v.y + e.y, v.z + e.z, v.w);
                }
            }
        }
        if (chunks <= warps) break;
        if (lane == 0u) c = atomicAdd(ctl + kExtFetch, 1u);
        c = warps + __shfl_sync(0xffffffffu, c, 0);
    }
    flush_tally(counters, tally, 0u, 0u);
}

// Persistent traversal with lane refill. Each lane walks its own ray
// (closest_step / any_step); once at least kRefill lanes of the warp are
// idle, the warp takes that many new rays from the queue in one atomic and
// hands them to the idle lanes, while the other lanes keep their walks.
// Finished rays write their results in the same refill round, so ray set-up
// and result stores run for the idle lanes together. kBurst steps run
// between two refill checks. Without refill, a warp that took 32 rays runs
// until the slowest of them ends. As many lanes of a warp take rays as
// rays_per_grab allows, and warps that the queue cannot reach leave before
// their first atomic (probe baker over 2,000 sites, 8 samples, in form 1: 5.24 -> 2.79 ms).
template <int kRefill, int kBurst, class Src>
__global__ void __launch_bounds__(128, 9) k_wf_extend_refill(Src src, const uint32_t* __restrict__ queue,
                                                          uint32_t* ctl, const float4* __restrict__ ro,
                                                          const float4* __restrict__ rd, float4* __restrict__ hit,
                                                          unsigned long long* counters) {
    const uint32_t count = *(volatile uint32_t*)(ctl + kExt);
    const uint32_t lane = threadIdx.x & 31u;
    const unsigned below = (1u << lane) - 1u;
    const uint32_t share = rays_per_grab(count);
    if ((uint64_t)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * share >= count) return;  // the whole warp
    const unsigned lanes = 0xffffffffu >> (32u - share);
    const int refill = min(kRefill, (int)share);
    RayTally tally{0u, 0u};
    ClosestWalk w;
    int stack[kTraversalStack];
    bool alive = false, pending = false, drained = false;
    uint32_t p = 0u;
    for (;;) {
        const unsigned idle = __ballot_sync(0xffffffffu, !alive) & lanes;
        if (drained) {
            if (idle == lanes) break;
        } else if (__popc(idle) >= refill) {
            if (pending) {
                const HitInfo h = closest_end(src.of(p), w);
                hit[p] = make_float4(__uint_as_float(h.valid ? h.flat : 0xffffffffu), h.t, h.b1, h.b2);
                pending = false;
            }
            const uint32_t n = (uint32_t)__popc(idle);
            uint32_t base = 0u;
            if (lane == 0u) base = atomicAdd(ctl + kExtFetch, n);
            base = __shfl_sync(0xffffffffu, base, 0);
            if ((idle >> lane) & 1u) {
                const uint32_t idx = base + (uint32_t)__popc(idle & below);
                if (idx < count) {
                    p = queue[idx];
                    const float4 o = ro[p], d = rd[p];
                    tally.extend++;
                    alive = closest_begin(src.of(p), w, xyz(o), xyz(d), o.w, d.w);
                    pending = !alive;
                }
            }
            if (base + n >= count) drained = true;
            continue;
        }
        if (alive) {
            const SceneView& s = src.of(p);
#pragma unroll 1
            for (int k = 0; k < kBurst; ++k) {
                if (!closest_step<kTraversalStack>(s, w, stack)) {
                    alive = false;
                    pending = true;
                    break;
                }
            }
        }
    }
    if (pending) {
        const HitInfo h = closest_end(src.of(p), w);
        hit[p] = make_float4(__uint_as_float(h.valid ? h.flat : 0xffffffffu), h.t, h.b1, h.b2);
    }
    flush_tally(counters, tally, 0u, 0u);
}

template <int kRefill, int kBurst, class Src>
__global__ void __launch_bounds__(128, 9) k_wf_shadow_refill(Src src, const float4* __restrict__ queue, uint32_t* ctl,
                                                          float t_max, float4* __restrict__ rad,
                                                          float4* __restrict__ si, unsigned long long* counters) {
    const uint32_t count = *(volatile uint32_t*)(ctl + kShd);
    const uint32_t lane = threadIdx.x & 31u;
    const unsigned below = (1u << lane) - 1u;
    const uint32_t share = rays_per_grab(count);
    if ((uint64_t)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * share >= count) return;  // the whole warp
    const unsigned lanes = 0xffffffffu >> (32u - share);
    const int refill = min(kRefill, (int)share);
    RayTally tally{0u, 0u};
    AnyWalk w;
    int stack[kTraversalStack];
    bool alive = false, pending = false, drained = false;
    uint32_t p = 0u, e = 0u;
    for (;;) {
        const unsigned idle = __ballot_sync(0xffffffffu, !alive) & lanes;
        if (drained) {
            if (idle == lanes) break;
        } else if (__popc(idle) >= refill) {
            if (pending) {  // a ray that ended without a hit adds its contribution
                const float4 b = queue[3u * e + 1u], c = queue[3u * e + 2u];
                float4* target = (__float_as_uint(b.w) == kKindNee) ? rad : si;
                const float4 v = target[p];
                target[p] = make_float4(v.x + c.x, v.y + c.y, v.z + c.z, v.w);
                pending = false;
            }
            const uint32_t n = (uint32_t)__popc(idle);
            uint32_t base = 0u;
            if (lane == 0u) base = atomicAdd(ctl + kShdFetch, n);
            base = __shfl_sync(0xffffffffu, base, 0);
            if ((idle >> lane) & 1u) {
                const uint32_t idx = base + (uint32_t)__popc(idle & below);
                if (idx < count) {
                    e = idx;
                    const float4 a = queue[3u * idx], b = queue[3u * idx + 1u], c = queue[3u * idx + 2u];
                    tally.shadow++;
                    p = __float_as_uint(a.w);
                    alive = any_begin(src.of(p), w, xyz(a), xyz(b), 0.0f, c.w > 0.0f ? c.w : t_max);
                    pending = !alive;
                }
            }
            if (base + n >= count) drained = true;
            continue;
        }
        if (alive) {
            const SceneView& s = src.of(p);
#pragma unroll 1
            for (int k = 0; k < kBurst; ++k) {
                const int r = any_step<kTraversalStack>(s, w, stack);
                if (r != 0) {
                    alive = false;
                    pending = r == 1;
                    break;
                }
            }
        }
    }
    if (pending) {
        const float4 b = queue[3u * e + 1u], c = queue[3u * e + 2u];
        float4* target = (__float_as_uint(b.w) == kKindNee) ? rad : si;
        const float4 v = target[p];
        target[p] = make_float4(v.x + c.x, v.y + c.y, v.z + c.z, v.w);
    }
    flush_tally(counters, tally, 0u, 0u);
}

// The path-state stages are bound by the latency of their gathers (scene
// records, path state) more than by bandwidth (10 long-scoreboard stalls an
// issue, 2.3 to 2.5 TB/s of DRAM traffic): 6 blocks of 128 per SM (80
// registers), the texel stage 8 (64 registers, 212 B of spills; 18.8 ms for
// the 200k texel iteration against 19.3 with 6).
// ---------------------------------------------------------------------------
// Texture-space integrator stages (texture_space_path_tracer.slang:57-216).
// ---------------------------------------------------------------------------
struct TexelArgs {
    McView mc;
    uint4* slots;
    uint32_t iteration;
    uint32_t n;  // samples per texel
    uint32_t max_bounces;
    int reset;
    // points mode (irradiance at given surface points instead of texels)
    const float4* points;  // (b1, b2, instance bits, primitive bits | back << 31)
    float4* point_out;     // (E rgb, 0), or (0, 0, 0, -1) for no point
    int indirect_only;     // points mode: leave out the direct sun irradiance term
};

// Start sample k of the current side: sun irradiance shadow ray (at its slot
// of the round's queue), first direction (estimate_surface_irradiance,
// texture_space_path_tracer.slang:95-113).
__device__ __forceinline__ PathNext texel_start_sample(const SceneView& s, const LightParams& L, const WfState& st,
                                                       const WfQueues& q, int buf, uint32_t shadow_slot, uint32_t p,
                                                       uint32_t flags, Rng& rng, bool direct) {
    const float4 sf = st.surf[p];
    const uint32_t inst = __float_as_uint(sf.z), prim = __float_as_uint(sf.w);
    f3 view = world_flat_normal(s, inst, prim);
    if (flags & kFlagBack) view = -view;
    const Shading sd = shading_data(s, inst, prim, sf.x, sf.y, view);
    const float u0 = rng.next_1d(), u1 = rng.next_1d();
    const f3 l = sample_cone_direction(L.sun_dir, L.cos_half, u0, u1);
    const float ndl = maxf(0.0f, dot3(sd.frame.n, l));
    // the two draws are taken either way, so the RNG streams stay aligned
    if (direct) store_shadow(q, buf, shadow_slot, p, sd.origin_front, l, L.illum * ndl, kKindSun);
    st.si[p] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    st.rad[p] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    st.thp[p] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
    const float e0 = rng.next_1d(), e1 = rng.next_1d();
    float pdf;
    const f3 dir = cosine_sample_hemisphere(e0, e1, &pdf);
    flags &= ~(kFlagNoPath | kBounceMask);
    const bool path = pdf > 1e-6f;
    if (path) {
        st.ro[p] = f4(sd.origin_front, 0.0f);
        st.rd[p] = f4(sd.frame.to_global(dir), L.t_max);
        st.zpdf[p] = make_float2(fabsf(dir.z), pdf);
    } else {
        flags |= kFlagNoPath;
    }
    st.flags[p] = flags;
    return path ? kWalk : kAwaitClose;
}

__global__ void __launch_bounds__(kStageThreads, 6) k_wf_texel_generate(SceneView s, LightingRaw lraw, TexelArgs a,
                                                                     WfState st, WfQueues q, uint32_t begin,
                                                                     uint32_t count, unsigned long long* counters) {
    __shared__ BlockAppend sh[2];
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    TexelSurface ts;
    Rng rng(0u, 0u, 0u);
    const bool unit = p < count && texel_surface(s, a.mc, begin + p, a.iteration, a.n, &ts, &rng);
    const bool two_sided = unit && (ts.side.y & 1u);
    const uint32_t slot = shadow_slots(sh[0], q.ctl, unit);
    PathNext next = kRetire;
    if (unit) {
        const LightParams L = make_light(lraw);
        st.unit[p] = begin + p;
        st.surf[p] = make_float4(ts.b1, ts.b2, __uint_as_float(ts.inst), __uint_as_float(ts.prim));
        st.irr[p] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        next = texel_start_sample(s, L, st, q, 1, slot, p, two_sided ? kFlagTwoSided : 0u, rng, true);
        st.rng[p] = rng.state;
    }
    push_paths(sh[1], q, 0, q.ctl + kCtlWords, p, next);
    count_units(counters, unit, two_sided ? 2u * a.n : a.n);
}

// Surface points instead of texels: the same estimator at the listed points,
// with RNG(index, 0xFFFFFFFF, iteration * n) and view = the flat normal,
// negated for the back side.
__global__ void __launch_bounds__(kStageThreads) k_wf_point_generate(SceneView s, LightingRaw lraw, TexelArgs a,
                                                                  WfState st, WfQueues q, uint32_t begin,
                                                                  uint32_t count, unsigned long long* counters) {
    __shared__ BlockAppend sh[2];
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t u = begin + p;
    float4 pt = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    bool unit = p < count;
    uint32_t inst = 0u, primw = 0u;
    if (unit) {
        pt = a.points[u];
        inst = __float_as_uint(pt.z);
        primw = __float_as_uint(pt.w);
        if (inst == 0xffffffffu || !valid_prim(s, inst, primw & 0x7fffffffu)) {
            if (inst != 0xffffffffu) atomicOr(s.status, kStatusBadRecord);
            a.point_out[u] = make_float4(0.0f, 0.0f, 0.0f, -1.0f);
            unit = false;
        }
    }
    const uint32_t slot = shadow_slots(sh[0], q.ctl, unit && !a.indirect_only);
    PathNext next = kRetire;
    if (unit) {
        const LightParams L = make_light(lraw);
        Rng rng(u, 0xffffffffu, a.iteration * a.n);
        st.unit[p] = u;
        st.surf[p] = make_float4(pt.x, pt.y, __uint_as_float(inst), __uint_as_float(primw & 0x7fffffffu));
        st.irr[p] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        next = texel_start_sample(s, L, st, q, 1, slot, p, (primw >> 31) ? kFlagBack : 0u, rng, !a.indirect_only);
        st.rng[p] = rng.state;
    }
    push_paths(sh[1], q, 0, q.ctl + kCtlWords, p, next);
    count_units(counters, unit, a.n);
}

// One bounce of trace_radiance (texture_space_path_tracer.slang:60-83) for the
// paths whose hit the trace found, and the closing of finished samples: si +=
// L*|z|/pdf, irr += si, next sample / side, or the running-mean store
// (texture_space_path_tracer.slang:111-138, 203-215).
__global__ void __launch_bounds__(kStageThreads, 8) k_wf_texel_stage(SceneView s, LightingRaw lraw, TexelArgs a,
                                                                  WfState st, WfQueues q, int buf, uint32_t* ctl) {
    __shared__ BlockAppend sh[2];
    const uint32_t walking = *(volatile uint32_t*)(ctl + kExt);
    const uint32_t count = walking + *(volatile uint32_t*)(ctl + kClose);
    const LightParams L = make_light(lraw);
    for (uint32_t base = blockIdx.x * blockDim.x; base < count; base += gridDim.x * blockDim.x) {
        const uint32_t idx = base + threadIdx.x;
        const bool live = idx < count;
        uint32_t p = 0u, flags = 0u, flat = 0xffffffffu;
        float4 h = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (live) {
            p = q.ext[buf][idx < walking ? idx : q.cap - 1u - (idx - walking)];
            flags = st.flags[p];
            if (idx < walking) {
                h = st.hit[p];
                flat = __float_as_uint(h.x);
            }
        }
        const bool at_hit = flat != 0xffffffffu;
        const bool more_samples = (flags >> kSampleShift) + 1u < a.n;
        const bool to_back = !more_samples && !a.point_out && !(flags & kFlagBack) && (flags & kFlagTwoSided);
        const bool starts = live && !at_hit && (more_samples || to_back);
        const uint32_t slot = shadow_slots(sh[0], ctl, at_hit || (starts && (to_back || !a.indirect_only)));
        PathNext next = kRetire;
        if (at_hit) {
            const f3 d = xyz(st.rd[p]);
            f3 thp = xyz(st.thp[p]), rad = xyz(st.rad[p]);
            Rng rng(0u, 0u, 0u);
            rng.state = st.rng[p];
            const uint2 ref = __ldg(s.tri_refs + flat);
            const Shading sd = shading_data(s, ref.x, ref.y, h.z, h.w, -d);
            rad = rad + thp * sd.emissive;
            const float u0 = rng.next_1d(), u1 = rng.next_1d();
            const f3 l = sample_cone_direction(L.sun_dir, L.cos_half, u0, u1);
            const float ndl = maxf(0.0f, dot3(sd.frame.n, l));
            const f3 f = sd.diffuse * kInvPi;
            store_shadow(q, buf, slot, p, sd.origin_front, l, thp * ((f * L.illum) * ndl), kKindNee);
            const float e0 = rng.next_1d(), e1 = rng.next_1d();
            float pdf;
            const f3 sdir = cosine_sample_hemisphere(e0, e1, &pdf);
            next = kAwaitClose;
            if (pdf > 1e-6f) {
                const uint32_t bounce = ((flags & kBounceMask) >> kBounceShift) + 1u;
                flags = (flags & ~kBounceMask) | (bounce << kBounceShift);
                if (bounce < a.max_bounces) {
                    next = kWalk;
                    thp = thp * ((f * fabsf(sdir.z)) / pdf);
                    st.ro[p] = f4(sd.origin_front, 0.0f);
                    st.rd[p] = f4(sd.frame.to_global(sdir), L.t_max);
                    st.thp[p] = f4(thp, 0.0f);
                }
            }
            st.rad[p] = f4(rad, 0.0f);
            st.rng[p] = rng.state;
            st.flags[p] = flags;
        } else if (live) {
            f3 si = xyz(st.si[p]);
            if (!(flags & kFlagNoPath)) {
                f3 rad = xyz(st.rad[p]);
                if (idx < walking) rad = rad + xyz(st.thp[p]) * sky_radiance(L, xyz(st.rd[p]));
                const float2 zp = st.zpdf[p];
                si = si + ((rad * zp.x) / zp.y);
            }
            f3 irr = xyz(st.irr[p]) + si;
            if (!more_samples) {
                const uint32_t u = st.unit[p];
                if (a.point_out) {
                    a.point_out[u] = f4(irr / (float)a.n, 0.0f);
                } else {
                    // side complete: running mean into its slot
                    const uint32_t inst = __float_as_uint(st.surf[p].z);
                    const uint4 info = __ldg(a.mc.instance_infos + inst);
                    const uint2 side = __ldg(a.mc.side_infos + inst);
                    const uint32_t global_texel = info.z + (u - __ldg(a.mc.surface_prefix + inst));
                    const uint32_t to = (flags & kFlagBack) ? side.x + (global_texel - info.z) : global_texel;
                    if (to < a.mc.payload_count)
                        store_running_mean(a.slots, to, irr / (float)a.n, a.reset, a.mc.compensation);
                    else
                        atomicOr(s.status, 2u);
                }
                irr = mk3(0.0f, 0.0f, 0.0f);
            }
            if (starts) {
                const uint32_t low = flags & ((1u << kSampleShift) - 1u);
                const uint32_t k = (flags >> kSampleShift) + 1u;
                st.irr[p] = f4(irr, 0.0f);
                Rng rng(0u, 0u, 0u);
                rng.state = st.rng[p];
                next = texel_start_sample(s, L, st, q, buf, slot, p, to_back ? (low | kFlagBack) : (low | (k << kSampleShift)),
                                          rng, to_back || !a.indirect_only);
                st.rng[p] = rng.state;
            }
        }
        push_paths(sh[1], q, buf ^ 1, ctl + kCtlWords, p, next);
    }
}


// ---------------------------------------------------------------------------
// Screen path tracer stages (path_tracer.slang:40-130, camera.slang:201-236).
// ---------------------------------------------------------------------------
struct CameraWf {  // layout of NanCamera
    float position[3];
    float jitter_x;
    float image_u[3];
    float jitter_y;
    float image_v[3];
    float near_clip;
    float image_w[3];
    float far_clip;
};

// Cached frames: paths end at their second hit, which becomes a cache query
// (position and pixel, shading normal, weight = throughput * albedo / pi).
// Pixels (offset + i * stride) mod P for i < train_count also record the
// hit as training point i.
struct CachedArgs {
    float4* queries;  // 2 per query
    float4* weights;
    uint32_t* query_count;
    float4* train_points;
    float4* train_queries;  // 2 per training point
    uint32_t train_count, train_offset, train_inverse;
    uint32_t vertex;  // path vertex that queries the cache: 0 (indirect) or 1
};

struct ScreenArgs {
    CameraWf cam;
    float4* out;
    uint32_t width, height, frame, max_vertices;
    int cached;
    CachedArgs cache;
};

__global__ void __launch_bounds__(kStageThreads) k_wf_screen_generate(SceneView s, LightingRaw lraw, ScreenArgs a, WfState st,
                                                            WfQueues q, uint32_t begin, uint32_t count,
                                                            unsigned long long* counters) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= count) return;
    const uint32_t pixel = begin + p;
    const uint32_t px = pixel % a.width, py = pixel / a.width;
    Rng rng(px, py, a.frame * 1u + 0u);
    rng.next_1d();
    rng.next_1d();  // the unused jitter draw (path_tracer.slang:121)
    const CameraWf& cam = a.cam;
    float pxf = ((float)px + 0.5f) / (float)a.width;
    float pyf = ((float)py + 0.5f) / (float)a.height;
    pxf = pxf + (-cam.jitter_x);
    pyf = pyf + cam.jitter_y;
    const float nx = 2.0f * pxf + -1.0f;
    const float ny = -2.0f * pyf + 1.0f;
    const f3 U = mk3(cam.image_u[0], cam.image_u[1], cam.image_u[2]);
    const f3 V = mk3(cam.image_v[0], cam.image_v[1], cam.image_v[2]);
    const f3 W = mk3(cam.image_w[0], cam.image_w[1], cam.image_w[2]);
    const f3 dir = normalize3((nx * U + ny * V) + W);
    const float inv_cos = 1.0f / dot3(normalize3(W), dir);
    st.unit[p] = pixel;
    st.rng[p] = rng.state;
    st.flags[p] = 0u;
    st.ro[p] = f4(mk3(cam.position[0], cam.position[1], cam.position[2]), cam.near_clip * inv_cos);
    st.rd[p] = f4(dir, cam.far_clip * inv_cos);
    st.thp[p] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
    st.rad[p] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    st.si[p] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    st.zpdf[p] = make_float2(0.0f, 1.0f);
    // every pixel of the chunk is a path: queue and counters need no appends
    q.ext[0][p] = p;
    if (p == 0u) {
        q.ctl[kCtlWords + kExt] = count;
        atomicAdd(counters + 2, (unsigned long long)count);
        atomicAdd(counters + 3, (unsigned long long)count);
    }
}

// The area-light term of the previous vertex (kept apart by the shadow stage)
// joins the radiance after that vertex's sun term, as in the loop's order.
__device__ __forceinline__ f3 fold_area_term(const WfState& st, uint32_t p, f3 rad) {
    const float4 a = st.si[p];
    st.si[p] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    return rad + xyz(a);
}

// Shades the hit of path p (path_tracer.slang:54-82); its sun ray goes to
// `slot` of the round's shadow queue.
__device__ __forceinline__ PathNext screen_shade_path(const SceneView& s, const LightParams& L, const ScreenArgs& a,
                                                      const WfState& st, const WfQueues& q, int buf, uint32_t* ctl,
                                                      uint32_t p, uint32_t flags, uint32_t vertex, float4 h,
                                                      bool at_cache, uint32_t slot) {
    const f3 d = xyz(st.rd[p]);
    f3 thp = xyz(st.thp[p]), rad = xyz(st.rad[p]);
    if (L.area_nee) rad = fold_area_term(st, p, rad);
    const uint32_t flat = __float_as_uint(h.x);
    Rng rng(0u, 0u, 0u);
    rng.state = st.rng[p];
    const uint2 ref = __ldg(s.tri_refs + flat);
    const Shading sd = shading_data(s, ref.x, ref.y, h.z, h.w, -d);
    if (L.area_nee && vertex > 0u)
        rad = rad + thp * (sd.emissive * area_mis_weight(s, sd.emissive, sd.face_normal, d, h.y, st.zpdf[p].y));
    else
        rad = rad + thp * sd.emissive;
    const f3 f = sd.diffuse * kInvPi;
    if (at_cache) {
        // the rest of the path is the cache's irradiance at this point;
        // at vertex 0 the sun is still sampled (NEE) and the cache holds
        // the indirect irradiance only
        if (vertex == 0u) {
            const float u0 = rng.next_1d(), u1 = rng.next_1d();
            const f3 l = sample_cone_direction(L.sun_dir, L.cos_half, u0, u1);
            const float ndl = maxf(0.0f, dot3(sd.frame.n, l));
            store_shadow(q, buf, slot, p, sd.origin_front, l, thp * ((f * L.illum) * ndl), kKindNee);
        }
        const uint32_t pixel = st.unit[p];
        const uint32_t qi = queue_slot(a.cache.query_count, true);
        const float4 q0 = make_float4(sd.position.x, sd.position.y, sd.position.z, __uint_as_float(pixel));
        const float4 q1 = f4(sd.frame.n, 0.0f);
        a.cache.queries[2u * qi] = q0;
        a.cache.queries[2u * qi + 1u] = q1;
        a.cache.weights[qi] = f4(thp * f, 0.0f);
        const uint32_t P = a.width * a.height;
        const uint32_t rel = pixel >= a.cache.train_offset ? pixel - a.cache.train_offset
                                                           : pixel + (P - a.cache.train_offset);
        const uint32_t ti = (uint32_t)(((uint64_t)rel * a.cache.train_inverse) % P);
        if (ti < a.cache.train_count) {
            // a back side exists for double-sided materials only (as texel back slots)
            const bool two = (__float_as_uint(__ldg(tri_refs(s, ref.x, ref.y).mat + 3)) & 1u) != 0u;
            const bool back = two && dot3(world_flat_normal(s, ref.x, ref.y), -d) < 0.0f;
            a.cache.train_points[ti] = make_float4(h.z, h.w, __uint_as_float(ref.x),
                                                   __uint_as_float(ref.y | (back ? 0x80000000u : 0u)));
            a.cache.train_queries[2u * ti] = q0;
            a.cache.train_queries[2u * ti + 1u] = q1;
        }
        if (vertex == 0u) {
            st.rad[p] = f4(rad, 0.0f);
            return kAwaitClose;  // its sun ray is in flight
        }
        if (L.area_nee) rad = rad + mk3(0.0f, 0.0f, 0.0f);
        a.out[pixel] = f4(rad, 1.0f);
        return kRetire;
    }
    const float u0 = rng.next_1d(), u1 = rng.next_1d();
    const f3 l = sample_cone_direction(L.sun_dir, L.cos_half, u0, u1);
    const float ndl = maxf(0.0f, dot3(sd.frame.n, l));
    store_shadow(q, buf, slot, p, sd.origin_front, l, thp * ((f * L.illum) * ndl), kKindNee);
    // light reached from this vertex lies on the next one: sampled only
    // where that vertex exists, so both strategies cover the same paths
    if (L.area_nee && vertex + 1u < a.max_vertices) {
        const float us = rng.next_1d(), a0 = rng.next_1d(), a1 = rng.next_1d();
        const AreaSample as = area_nee_sample(s, sd, us, a0, a1);
        if (as.valid)
            store_shadow(q, buf, queue_slot(ctl + kShd, true), p, sd.origin_front, as.dir, thp * as.contrib, kKindSun,
                         as.tmax);
    }
    const float e0 = rng.next_1d(), e1 = rng.next_1d();
    float pdf;
    const f3 wo = cosine_sample_hemisphere(e0, e1, &pdf);
    pdf = maxf(pdf, 1e-6f);
    st.zpdf[p] = make_float2(0.0f, pdf);
    thp = thp * ((f * fabsf(wo.z)) / pdf);
    st.ro[p] = f4(sd.origin_front, 0.0f);
    st.rd[p] = f4(sd.frame.to_global(wo), L.t_max);
    const uint32_t next = vertex + 1u;
    st.thp[p] = f4(thp, 0.0f);
    st.rad[p] = f4(rad, 0.0f);
    st.rng[p] = rng.state;
    st.flags[p] = (flags & ~kBounceMask) | (next << kBounceShift);
    return next >= a.max_vertices ? kAwaitClose : kWalk;
}

__global__ void __launch_bounds__(kStageThreads, 6) k_wf_screen_stage(SceneView s, LightingRaw lraw, ScreenArgs a,
                                                                   WfState st, WfQueues q, int buf, uint32_t* ctl) {
    __shared__ BlockAppend sh[2];
    const uint32_t walking = *(volatile uint32_t*)(ctl + kExt);
    const uint32_t count = walking + *(volatile uint32_t*)(ctl + kClose);
    const LightParams L = make_light(lraw);
    for (uint32_t base = blockIdx.x * blockDim.x; base < count; base += gridDim.x * blockDim.x) {
        const uint32_t idx = base + threadIdx.x;
        const bool live = idx < count;
        uint32_t p = 0u, flags = 0u, flat = 0xffffffffu;
        float4 h = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (live) p = q.ext[buf][idx < walking ? idx : q.cap - 1u - (idx - walking)];
        if (idx < walking) {
            flags = st.flags[p];
            h = st.hit[p];
            flat = __float_as_uint(h.x);
        }
        const uint32_t vertex = (flags & kBounceMask) >> kBounceShift;
        const bool at_hit = flat != 0xffffffffu;
        const bool at_cache = at_hit && a.cached && vertex == a.cache.vertex;
        const uint32_t slot = shadow_slots(sh[0], ctl, at_hit && !(at_cache && vertex > 0u));
        PathNext next = kRetire;
        if (at_hit) {
            next = screen_shade_path(s, L, a, st, q, buf, ctl, p, flags, vertex, h, at_cache, slot);
        } else if (live) {
            f3 rad = xyz(st.rad[p]);
            // the last vertex's area-light term follows its sun term
            if (L.area_nee) rad = rad + xyz(st.si[p]);
            if (idx < walking) {
                const f3 d = xyz(st.rd[p]);
                f3 sky = sky_radiance(L, d);
                if (vertex == 0u && L.sun_disk) sky = sky + sun_disk(L, d);
                rad = rad + xyz(st.thp[p]) * sky;
                if (L.area_nee) rad = rad + mk3(0.0f, 0.0f, 0.0f);
            }
            a.out[st.unit[p]] = f4(rad, 1.0f);
        }
        push_paths(sh[1], q, buf ^ 1, ctl + kCtlWords, p, next);
    }
}

// ---------------------------------------------------------------------------
// Surface-probe baker stages (surface_probe_path_tracer.slang:151-315).
// ---------------------------------------------------------------------------
struct ProbeArgs {
    ProbeOut out;
    const float4* probes;
    const float4* pinst;
    uint32_t probe_instance_count;
    uint32_t iteration, n, spp, max_bounces;
    int reset;
};

// Shading of the probe's own surface point (estimate_surface_irradiance).
__device__ __forceinline__ Shading probe_surface(const SceneView& s, const ProbeArgs& a, uint32_t probe,
                                                 const float4& surf) {
    const float4 nrm = __ldg(a.probes + 3u * probe + 1u);
    const f3 view = normalize3(mk3(nrm.x, nrm.y, nrm.z));
    return shading_data(s, __float_as_uint(surf.z), __float_as_uint(surf.w), surf.x, surf.y, view);
}

// One cosine sample around the face normal (no sun at the probe itself).
__device__ __forceinline__ PathNext probe_start_sample(const SceneView& s, const LightParams& L, const ProbeArgs& a,
                                                       const WfState& st, uint32_t p, uint32_t flags, Rng& rng) {
    const float4 surf = st.surf[p];
    const Shading sd = probe_surface(s, a, st.unit[p], surf);
    const float kr = st.si[p].w;
    const float e0 = rng.next_1d(), e1 = rng.next_1d();
    float pdf;
    const f3 dir = cosine_sample_hemisphere(e0, e1, &pdf);
    flags &= ~(kFlagNoPath | kBounceMask);
    if (pdf > 1e-6f) {
        const f3 o = sd.origin_front;
        st.ro[p] = f4(o, 0.0f);
        st.rd[p] = f4(Frame(normalize3(sd.face_normal)).to_global(dir), L.t_max);
        st.thp[p] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
        st.rad[p] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        st.zpdf[p] = make_float2(fabsf(dir.z), pdf);
        st.pa[p] = make_float4(surf.z, surf.w, len3(o - sd.position), 2.0f * kr);
        uint4 b = st.pb[p];
        b.x = 0u;
        b.w = radial_texel(dir);
        st.pb[p] = b;
    } else {
        flags |= kFlagNoPath;
    }
    st.flags[p] = flags;
    return (flags & kFlagNoPath) ? kAwaitClose : kWalk;
}

// Per-path bodies of the probe stages, shared by the one-scene kernels and the
// multi-scene batch kernels (which look up the path's probe set first).
__device__ __forceinline__ PathNext probe_generate_path(const SceneView& s, const LightParams& L, const ProbeArgs& a,
                                                        const WfState& st, uint32_t probe, uint32_t p) {
    const uint4 meta = __ldg(reinterpret_cast<const uint4*>(a.probes) + 3u * probe + 2u);
    const uint32_t inst = meta.w >> 8;
    if (inst >= a.probe_instance_count || !valid_prim(s, inst, meta.x)) {
        atomicOr(s.status, kStatusBadRecord);
        return kRetire;
    }
    const float4 params = __ldg(a.pinst + 3u * inst + 2u);
    st.unit[p] = probe;
    st.surf[p] = make_float4(__uint_as_float(meta.y), __uint_as_float(meta.z), __uint_as_float(inst),
                             __uint_as_float(meta.x));
    st.si[p] = make_float4(0.0f, 0.0f, 0.0f, maxf(params.x, 1e-6f));
    st.irr[p] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const uint32_t prev_iter = a.reset ? 0u : a.out.counts[probe];
    st.pb[p] = make_uint4(0u, 0u, prev_iter, 0u);
    st.pc[2u * p] = make_uint4(0u, 0u, 0u, 0u);
    st.pc[2u * p + 1u] = make_uint4(0u, 0u, 0u, 0u);
    if (a.reset)
        for (int t = 0; t < 16; ++t) a.out.radial[16u * probe + (uint32_t)t] = 0u;
    Rng rng(probe, inst, a.iteration * a.n);
    const PathNext next = probe_start_sample(s, L, a, st, p, 0u, rng);
    st.rng[p] = rng.state;
    return next;
}

// The path leaves the scene: its sample can be closed.
__device__ __forceinline__ void probe_miss_path(const LightParams& L, const WfState& st, uint32_t p) {
    const uint32_t bounce = (st.flags[p] & kBounceMask) >> kBounceShift;
    if (bounce == 0u) {
        float4 pa = st.pa[p];
        pa.w = 2.0f * st.si[p].w;
        st.pa[p] = pa;
    }
    st.rad[p] = f4(xyz(st.rad[p]) + xyz(st.thp[p]) * sky_radiance(L, xyz(st.rd[p])), 0.0f);
}

// Shades the path's hit; its sun ray goes to `slot` of the round's shadow
// queue.
__device__ __forceinline__ PathNext probe_shade_path(const SceneView& s, const LightParams& L, const ProbeArgs& a,
                                                     const WfState& st, const WfQueues& q, int buf, uint32_t slot,
                                                     uint32_t p, float4 h) {
    uint32_t flags = st.flags[p];
    const f3 d = xyz(st.rd[p]);
    f3 thp = xyz(st.thp[p]), rad = xyz(st.rad[p]);
    float4 pa = st.pa[p];  // src inst, src prim, src offset, first hit
    const uint32_t bounce = (flags & kBounceMask) >> kBounceShift;
    const float radial_max = 2.0f * st.si[p].w;
    const uint32_t flat = __float_as_uint(h.x);
    if (bounce == 0u) pa.w = minf(h.y, radial_max);
    const uint2 ref = __ldg(s.tri_refs + flat);
    const uint32_t src_inst = __float_as_uint(pa.x), src_prim = __float_as_uint(pa.y);
    const bool same_prim = ref.x == src_inst && ref.y == src_prim;
    const float thr = maxf(4.0f * pa.z, 1e-6f);
    const bool adjacent = ref.x == src_inst && h.y <= thr;
    if (same_prim || adjacent) {
        uint4 b = st.pb[p];
        b.x += 1u;
        st.pb[p] = b;
    }
    Rng rng(0u, 0u, 0u);
    rng.state = st.rng[p];
    const Shading sd = shading_data(s, ref.x, ref.y, h.z, h.w, -d);
    rad = rad + thp * sd.emissive;
    const float u0 = rng.next_1d(), u1 = rng.next_1d();
    const f3 l = sample_cone_direction(L.sun_dir, L.cos_half, u0, u1);
    const float ndl = maxf(0.0f, dot3(sd.frame.n, l));
    const f3 f = sd.diffuse * kInvPi;
    // the set's own t_max travels with the shadow ray (the batch mixes scenes)
    store_shadow(q, buf, slot, p, sd.origin_front, l, thp * ((f * L.illum) * ndl), kKindNee, L.t_max);
    const float e0 = rng.next_1d(), e1 = rng.next_1d();
    float pdf;
    const f3 sdir = cosine_sample_hemisphere(e0, e1, &pdf);
    bool ended = true;
    if (pdf > 1e-6f) {
        thp = thp * ((f * fabsf(sdir.z)) / pdf);
        const f3 next_origin = sd.origin_front;
        st.ro[p] = f4(next_origin, 0.0f);
        st.rd[p] = f4(Frame(normalize3(sd.face_normal)).to_global(sdir), L.t_max);
        pa.x = __uint_as_float(ref.x);
        pa.y = __uint_as_float(ref.y);
        pa.z = len3(next_origin - sd.position);
        const uint32_t next = bounce + 1u;
        flags = (flags & ~kBounceMask) | (next << kBounceShift);
        ended = next >= a.max_bounces;
    }
    st.pa[p] = pa;
    st.thp[p] = f4(thp, 0.0f);
    st.rad[p] = f4(rad, 0.0f);
    st.rng[p] = rng.state;
    st.flags[p] = flags;
    return ended ? kAwaitClose : kWalk;
}

// Closes the path's sample: the next one starts, or the probe's running mean
// is stored.
__device__ __forceinline__ PathNext probe_close_path(const SceneView& s, const LightParams& L, const ProbeArgs& a,
                                                     const WfState& st, uint32_t p) {
    const uint32_t flags = st.flags[p];
    const uint32_t probe = st.unit[p];
    f3 irr = xyz(st.irr[p]);
    uint4 b = st.pb[p];
    if (!(flags & kFlagNoPath)) {
        b.y += b.x;  // self-hit suspects of this sample
        const uint32_t texel = b.w;
        uint4 c = st.pc[2u * p + (texel >> 3)];
        const uint32_t word = (texel >> 1) & 3u, shift = (texel & 1u) * 16u;
        uint32_t* cw = word == 0u ? &c.x : (word == 1u ? &c.y : (word == 2u ? &c.z : &c.w));
        const uint32_t local = ((*cw >> shift) & 0xffffu) + 1u;
        *cw = (*cw & ~(0xffffu << shift)) | ((local & 0xffffu) << shift);
        st.pc[2u * p + (texel >> 3)] = c;
        const float kr = st.si[p].w;
        accumulate_radial_moment(a.out.radial, probe, texel, st.pa[p].w / maxf(kr, 1e-6f), b.z, local, a.spp);
        const float2 zp = st.zpdf[p];
        irr = irr + ((xyz(st.rad[p]) * zp.x) / zp.y);
    }
    st.pb[p] = b;
    const uint32_t k = (flags >> kSampleShift) + 1u;
    if (k < a.n) {
        st.irr[p] = f4(irr, 0.0f);
        Rng rng(0u, 0u, 0u);
        rng.state = st.rng[p];
        const PathNext next =
            probe_start_sample(s, L, a, st, p, (flags & ((1u << kSampleShift) - 1u)) | (k << kSampleShift), rng);
        st.rng[p] = rng.state;
        return next;
    }
    irr = irr / (float)a.n;
    const uint32_t prev = a.reset ? 0u : a.out.counts[probe];
    f3 pv = mk3(0.0f, 0.0f, 0.0f);
    if (prev != 0u)
        pv = mk3(a.out.values[3u * probe], a.out.values[3u * probe + 1u], a.out.values[3u * probe + 2u]);
    float4 comp = a.out.compensation ? a.out.compensation[probe] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const f3 acc = running_mean_step(pv, irr, prev, a.out.compensation ? &comp : nullptr);
    if (a.out.compensation) a.out.compensation[probe] = comp;
    a.out.values[3u * probe] = acc.x;
    a.out.values[3u * probe + 1u] = acc.y;
    a.out.values[3u * probe + 2u] = acc.z;
    a.out.counts[probe] = min(prev + 1u, 65535u);
    const uint32_t prev_self = a.reset ? 0u : a.out.self_hits[probe];
    a.out.self_hits[probe] = prev_self + b.y;
    return kRetire;
}

// A block's entry of a round's queue: its path and, while it walks, the hit
// the trace found.
struct StageEntry {
    uint32_t p;
    float4 hit;
    bool live, walks, at_hit;
};

__device__ __forceinline__ StageEntry stage_entry(const WfState& st, const WfQueues& q, int buf, uint32_t walking,
                                                  uint32_t count, uint32_t idx) {
    StageEntry e;
    e.live = idx < count;
    e.walks = idx < walking;
    e.p = 0u;
    e.hit = make_float4(__uint_as_float(0xffffffffu), 0.0f, 0.0f, 0.0f);
    if (e.live) e.p = q.ext[buf][e.walks ? idx : q.cap - 1u - (idx - walking)];
    if (e.walks) e.hit = st.hit[e.p];
    e.at_hit = __float_as_uint(e.hit.x) != 0xffffffffu;
    return e;
}

__global__ void __launch_bounds__(kStageThreads) k_wf_probe_generate(SceneView s, LightingRaw lraw, ProbeArgs a,
                                                                  WfState st, WfQueues q, uint32_t begin,
                                                                  uint32_t count, unsigned long long* counters) {
    __shared__ BlockAppend sh;
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    PathNext next = kRetire;
    if (p < count) next = probe_generate_path(s, make_light(lraw), a, st, begin + p, p);
    push_paths(sh, q, 0, q.ctl + kCtlWords, p, next);
    count_units(counters, next != kRetire, a.n);
}

__global__ void __launch_bounds__(kStageThreads, 6) k_wf_probe_stage(SceneView s, LightingRaw lraw, ProbeArgs a,
                                                                  WfState st, WfQueues q, int buf, uint32_t* ctl) {
    __shared__ BlockAppend sh[2];
    const uint32_t walking = *(volatile uint32_t*)(ctl + kExt);
    const uint32_t count = walking + *(volatile uint32_t*)(ctl + kClose);
    const LightParams L = make_light(lraw);
    for (uint32_t base = blockIdx.x * blockDim.x; base < count; base += gridDim.x * blockDim.x) {
        const StageEntry e = stage_entry(st, q, buf, walking, count, base + threadIdx.x);
        const uint32_t slot = shadow_slots(sh[0], ctl, e.at_hit);
        PathNext next = kRetire;
        if (e.at_hit) {
            next = probe_shade_path(s, L, a, st, q, buf, slot, e.p, e.hit);
        } else if (e.live) {
            if (e.walks) probe_miss_path(L, st, e.p);
            next = probe_close_path(s, L, a, st, e.p);
        }
        push_paths(sh[1], q, buf ^ 1, ctl + kCtlWords, e.p, next);
    }
}

// ---------------------------------------------------------------------------
// Multi-scene probe batch on the wavefront: every (set, probe) unit of the
// batch is one path in flight; each stage looks up the path's set (scene,
// lighting, records, outputs). The iteration and reset come from the batch's
// device control block, so a captured frame replays with the next iteration.
// ---------------------------------------------------------------------------
struct BatchWfArgs {
    const BatchSet* sets;
    const uint32_t* prefix;
    const BatchCtl* ctl;
    uint32_t* set_of;
    uint32_t set_count, total, n, spp, max_bounces;
    // independent samples: units [unit_begin, unit_begin + units) of this
    // chunk, one path per (unit, sample), and the per-sample results
    uint32_t unit_begin, units;
    ProbeSample* samples;
};

__device__ __forceinline__ uint32_t batch_set_of_unit(const BatchWfArgs& m, uint32_t u) {
    uint32_t lo = 0u, hi = m.set_count - 1u;  // set = last s with prefix[s] <= u
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1u) >> 1;
        if (__ldg(m.prefix + mid) <= u) lo = mid;
        else hi = mid - 1u;
    }
    return lo;
}

__device__ __forceinline__ ProbeArgs batch_probe_args(const BatchWfArgs& m, const BatchSet& b) {
    ProbeArgs a;
    a.out = b.out;
    a.probes = b.probes;
    a.pinst = b.pinst;
    a.probe_instance_count = b.probe_instance_count;
    a.iteration = m.ctl->iteration;
    a.n = m.n;
    a.spp = m.spp;
    a.max_bounces = m.max_bounces;
    a.reset = m.ctl->reset ? 1 : 0;
    return a;
}

__global__ void __launch_bounds__(kStageThreads) k_wfb_probe_generate(BatchWfArgs m, WfState st, WfQueues q,
                                                                   unsigned long long* counters) {
    __shared__ BlockAppend sh;
    const uint32_t u = blockIdx.x * blockDim.x + threadIdx.x;
    PathNext next = kRetire;
    if (u < m.total) {
        const uint32_t set = batch_set_of_unit(m, u);
        m.set_of[u] = set;
        const BatchSet& b = m.sets[set];
        next = probe_generate_path(b.s, make_light(b.light), batch_probe_args(m, b), st, u - __ldg(m.prefix + set), u);
    }
    push_paths(sh, q, 0, q.ctl + kCtlWords, u, next);
    count_units(counters, next != kRetire, m.n);
}

// Independent samples (NAN_BATCH_WAVEFRONT_INDEPENDENT): sample k of a probe
// draws from RNG(probe, instance, iteration * n + k) and is its own path, so a
// frame is max_bounces rounds and one that closes; every finished path stores
// its sample, and a last pass folds each probe's samples in sample order, as
// the independent-sample persistent kernel does.
__device__ __forceinline__ PathNext independent_generate_path(const BatchWfArgs& m, const WfState& st, uint32_t p) {
    const uint32_t uoff = p / m.n, k = p - uoff * m.n;
    const uint32_t u = m.unit_begin + uoff;
    const uint32_t set = batch_set_of_unit(m, u);
    m.set_of[p] = set;
    const BatchSet& b = m.sets[set];
    const uint32_t probe = u - __ldg(m.prefix + set);
    const ProbeArgs a = batch_probe_args(m, b);
    const uint4 meta = __ldg(reinterpret_cast<const uint4*>(a.probes) + 3u * probe + 2u);
    const uint32_t inst = meta.w >> 8;
    if (inst >= a.probe_instance_count || !valid_prim(b.s, inst, meta.x)) {
        atomicOr(b.s.status, kStatusBadRecord);
        ProbeSample none;
        none.si = mk3(0.0f, 0.0f, 0.0f);
        none.self_hits = 0u;
        none.texel = 0u;
        none.nd = 0.0f;
        none.has_path = false;
        m.samples[p] = none;
        return kRetire;
    }
    const float4 params = __ldg(a.pinst + 3u * inst + 2u);
    st.unit[p] = probe;
    st.surf[p] = make_float4(__uint_as_float(meta.y), __uint_as_float(meta.z), __uint_as_float(inst),
                             __uint_as_float(meta.x));
    st.si[p] = make_float4(0.0f, 0.0f, 0.0f, maxf(params.x, 1e-6f));
    st.pb[p] = make_uint4(0u, 0u, 0u, 0u);
    Rng rng(probe, inst, a.iteration * m.n + k);
    const PathNext next = probe_start_sample(b.s, make_light(b.light), a, st, p, 0u, rng);
    st.rng[p] = rng.state;
    return next;
}

__global__ void __launch_bounds__(kStageThreads) k_wfi_probe_generate(BatchWfArgs m, WfState st, WfQueues q) {
    __shared__ BlockAppend sh;
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    PathNext next = kRetire;
    if (p < m.units * m.n) next = independent_generate_path(m, st, p);
    push_paths(sh, q, 0, q.ctl + kCtlWords, p, next);
}

__global__ void __launch_bounds__(kStageThreads, 6) k_wfi_probe_stage(BatchWfArgs m, WfState st, WfQueues q, int buf,
                                                                   uint32_t* ctl) {
    __shared__ BlockAppend sh[2];
    const uint32_t walking = *(volatile uint32_t*)(ctl + kExt);
    const uint32_t count = walking + *(volatile uint32_t*)(ctl + kClose);
    for (uint32_t base = blockIdx.x * blockDim.x; base < count; base += gridDim.x * blockDim.x) {
        const StageEntry e = stage_entry(st, q, buf, walking, count, base + threadIdx.x);
        const uint32_t slot = shadow_slots(sh[0], ctl, e.at_hit);
        PathNext next = kRetire;
        if (e.live) {
            const uint32_t p = e.p;
            const BatchSet& b = m.sets[m.set_of[p]];
            if (e.at_hit) {
                next = probe_shade_path(b.s, make_light(b.light), batch_probe_args(m, b), st, q, buf, slot, p, e.hit);
            } else {
                if (e.walks) probe_miss_path(make_light(b.light), st, p);
                ProbeSample r;
                r.si = mk3(0.0f, 0.0f, 0.0f);
                r.self_hits = 0u;
                r.texel = 0u;
                r.nd = 0.0f;
                r.has_path = !(st.flags[p] & kFlagNoPath);
                if (r.has_path) {
                    const uint4 pb = st.pb[p];
                    const float2 zp = st.zpdf[p];
                    r.si = r.si + ((xyz(st.rad[p]) * zp.x) / zp.y);
                    r.self_hits = pb.x;
                    r.texel = pb.w;
                    r.nd = st.pa[p].w / maxf(st.si[p].w, 1e-6f);
                }
                m.samples[p] = r;
            }
        }
        push_paths(sh[1], q, buf ^ 1, ctl + kCtlWords, e.p, next);
    }
}

__global__ void __launch_bounds__(128) k_wfi_probe_fold(BatchWfArgs m, unsigned long long* counters) {
    const uint32_t uoff = blockIdx.x * blockDim.x + threadIdx.x;
    if (uoff >= m.units) return;
    const uint32_t u = m.unit_begin + uoff;
    const uint32_t set = batch_set_of_unit(m, u);
    const BatchSet& b = m.sets[set];
    const uint32_t probe = u - __ldg(m.prefix + set);
    const uint4 meta = __ldg(reinterpret_cast<const uint4*>(b.probes) + 3u * probe + 2u);
    const uint32_t inst = meta.w >> 8;
    if (inst >= b.probe_instance_count || !valid_prim(b.s, inst, meta.x)) return;
    const int reset = m.ctl->reset ? 1 : 0;
    const uint32_t prev_iter = reset ? 0u : b.out.counts[probe];
    if (reset)
        for (int t = 0; t < 16; ++t) b.out.radial[16u * probe + (uint32_t)t] = 0u;
    ProbeAcc acc;
    probe_acc_init(acc);
    for (uint32_t k = 0; k < m.n; ++k) probe_fold(acc, b.out, probe, m.samples[uoff * m.n + k], prev_iter, m.spp);
    probe_store(b.out, probe, acc, m.n, reset);
    RayTally none{0u, 0u};
    flush_tally(counters, none, 1u, m.n);
}

__global__ void __launch_bounds__(kStageThreads, 6) k_wfb_probe_stage(BatchWfArgs m, WfState st, WfQueues q, int buf,
                                                                   uint32_t* ctl) {
    __shared__ BlockAppend sh[2];
    const uint32_t walking = *(volatile uint32_t*)(ctl + kExt);
    const uint32_t count = walking + *(volatile uint32_t*)(ctl + kClose);
    for (uint32_t base = blockIdx.x * blockDim.x; base < count; base += gridDim.x * blockDim.x) {
        const StageEntry e = stage_entry(st, q, buf, walking, count, base + threadIdx.x);
        const uint32_t slot = shadow_slots(sh[0], ctl, e.at_hit);
        PathNext next = kRetire;
        if (e.live) {
            const BatchSet& b = m.sets[m.set_of[e.p]];
            const LightParams L = make_light(b.light);
            const ProbeArgs a = batch_probe_args(m, b);
            if (e.at_hit) {
                next = probe_shade_path(b.s, L, a, st, q, buf, slot, e.p, e.hit);
            } else {
                if (e.walks) probe_miss_path(L, st, e.p);
                next = probe_close_path(b.s, L, a, st, e.p);
            }
        }
        push_paths(sh[1], q, buf ^ 1, ctl + kCtlWords, e.p, next);
    }
}

LightingRaw to_raw(const NanLighting* l) {
    LightingRaw r;
    memcpy(&r, l, sizeof(r));
    return r;
}

SceneView scene_view(const NanContext* ctx) {
    SceneView v;
    v.nodes = ctx->nodes;
    v.tris = ctx->tris;
    const bool wide = ctx->wide_built && ctx->wnodes != nullptr && ctx->tuning.bvh_width == 8;
    v.wnodes = wide ? ctx->wnodes : nullptr;
    v.wtris = wide ? ctx->wtris : nullptr;
    v.tri_refs = ctx->tri_refs;
    v.vertices = ctx->scene.vertices;
    v.indices = ctx->scene.indices;
    v.mesh_descs = reinterpret_cast<const uint4*>(ctx->scene.mesh_descs);
    v.instance_descs = reinterpret_cast<const uint4*>(ctx->scene.instance_descs);
    v.transforms = ctx->scene.transforms;
    v.inverse_transposes = ctx->scene.inverse_transposes;
    v.materials = ctx->scene.materials;
    v.root = ctx->root;
    v.tri_count = ctx->tri_count;
    v.instance_count = ctx->scene.instance_count;
    v.status = ctx->d_status;
    v.lights = reinterpret_cast<const float4*>(ctx->lights);
    v.light_count = ctx->lights ? ctx->light_count : 0u;
    v.light_power = ctx->light_power;
    return v;
}

template <class T> T* carve(unsigned char*& cur, size_t count) {
    T* p = reinterpret_cast<T*>(cur);
    cur += ((count * sizeof(T) + 255u) / 256u) * 256u;
    return p;
}

// Traversal launches of one wavefront round: node width from the scene,
// the traversal form from the context's tuning (NanTuning.traversal).
template <class Src>
void launch_extend(const NanContext* ctx, int blocks, cudaStream_t st, bool wide, Src src, const uint32_t* queue,
                   uint32_t* ctl, const WfState& S) {
#define NAN_EXT_ARGS src, queue, ctl, S.ro, S.rd, S.hit, ctx->d_counters
    if (wide) k_wf_extend<8><<<blocks, 128, 0, st>>>(NAN_EXT_ARGS);
    else switch (ctx->tuning.traversal) {
        case 1: k_wf_extend_refill<8, 1, Src><<<blocks, 128, 0, st>>>(NAN_EXT_ARGS); break;
        case 2: k_wf_extend_refill<16, 1, Src><<<blocks, 128, 0, st>>>(NAN_EXT_ARGS); break;
        case 3: k_wf_extend_refill<24, 1, Src><<<blocks, 128, 0, st>>>(NAN_EXT_ARGS); break;
        case 4: k_wf_extend_refill<16, 4, Src><<<blocks, 128, 0, st>>>(NAN_EXT_ARGS); break;
        case 5: k_wf_extend<2, Src, 16><<<blocks, 128, 0, st>>>(NAN_EXT_ARGS); break;
        case 6: k_wf_extend<2, Src, 0, true><<<blocks, 128, 0, st>>>(NAN_EXT_ARGS); break;
        default: k_wf_extend<2><<<blocks, 128, 0, st>>>(NAN_EXT_ARGS); break;
    }
#undef NAN_EXT_ARGS
}

template <class Src>
void launch_shadow(const NanContext* ctx, int blocks, cudaStream_t st, bool wide, Src src, const float4* queue,
                   uint32_t* ctl, float t_max, const WfState& S) {
#define NAN_SHD_ARGS src, queue, ctl, t_max, S.rad, S.si, ctx->d_counters
    if (wide) k_wf_shadow<8><<<blocks, 128, 0, st>>>(NAN_SHD_ARGS);
    else switch (ctx->tuning.traversal) {
        case 1: k_wf_shadow_refill<8, 1, Src><<<blocks, 128, 0, st>>>(NAN_SHD_ARGS); break;
        case 2: k_wf_shadow_refill<16, 1, Src><<<blocks, 128, 0, st>>>(NAN_SHD_ARGS); break;
        case 3: k_wf_shadow_refill<24, 1, Src><<<blocks, 128, 0, st>>>(NAN_SHD_ARGS); break;
        case 4: k_wf_shadow_refill<16, 4, Src><<<blocks, 128, 0, st>>>(NAN_SHD_ARGS); break;
        case 5: k_wf_shadow<2, Src, 16><<<blocks, 128, 0, st>>>(NAN_SHD_ARGS); break;
        case 6: k_wf_shadow<2, Src, 0, true><<<blocks, 128, 0, st>>>(NAN_SHD_ARGS); break;
        default: k_wf_shadow<2><<<blocks, 128, 0, st>>>(NAN_SHD_ARGS); break;
    }
#undef NAN_SHD_ARGS
}

struct Grid {
    int persistent_blocks;
    int stream_blocks;
};

// Launch shapes for up to `paths` paths in flight: no more blocks than they
// can fill (a warp takes at least one ray of the at most three per path).
Grid grid_for(const NanContext* ctx, uint64_t paths) {
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
    int occ = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_wf_trace<2, OneScene>, 128, 0);
    Grid g;
    const int per_sm = ctx->tuning.trace_blocks_per_sm ? (int)ctx->tuning.trace_blocks_per_sm : std::max(occ, 1);
    g.persistent_blocks = (int)std::min<uint64_t>((uint64_t)sms * per_sm, std::max<uint64_t>((3 * paths + 3) / 4, 1));
    // 24 a SM are whole waves of the stages' 6 and 8 resident blocks: 16-scene probe
    // batch 14.10 -> 13.97 ms against 16 a SM (48: 14.01), other passes equal.
    g.stream_blocks = (int)std::min<uint64_t>((uint64_t)sms * 24, std::max<uint64_t>((paths + kStageThreads - 1) / kStageThreads, 1));
    return g;
}

// The traversal of round `it`: the closest hits of its walking paths and the
// shadow rays that the round before queued, in one launch; in two (extend, then
// shadow) for the traversal forms that refill lanes and for stage timing.
// timed: the pass is one that NanTuning.kernel_timing covers. The batch is not:
// its frames are captured in graphs, whose event records cannot be read.
// Launches apart leave out the queues that are empty by the plan: no path
// walks in the last of the rounds, and in the first there are shadow rays only
// if the generated paths have them (gen_shadows).
template <class Src>
void launch_trace(NanContext* ctx, int blocks, cudaStream_t st, bool wide, bool timed, bool gen_shadows, Src src,
                  const WfQueues& q, uint32_t it, uint32_t rounds, float t_max, const WfState& S) {
    const int buf = (int)(it & 1u);
    uint32_t* ctl = q.ctl + kCtlWords * (it + 1u);
    timed = timed && ctx->tuning.kernel_timing;
    const uint32_t form = wide ? 0u : ctx->tuning.traversal;
    if (!timed && (form == 0u || form >= 5u)) {
#define NAN_TRACE_ARGS src, q.ext[buf], ctl, S.ro, S.rd, S.hit, q.shd[buf ^ 1], ctl - kCtlWords, t_max, S.rad, S.si, \
                       ctx->d_counters
        if (wide) k_wf_trace<8, Src><<<blocks, 128, 0, st>>>(NAN_TRACE_ARGS);
        else if (form == 5u) k_wf_trace<2, Src, 16><<<blocks, 128, 0, st>>>(NAN_TRACE_ARGS);
        else if (form == 6u) k_wf_trace<2, Src, 0, true><<<blocks, 128, 0, st>>>(NAN_TRACE_ARGS);
        else k_wf_trace<2, Src><<<blocks, 128, 0, st>>>(NAN_TRACE_ARGS);
#undef NAN_TRACE_ARGS
        ctx->launches++;
        return;
    }
    if (it + 1u < rounds) {
        cudaEvent_t ev = timed ? nan_host::timing_begin(ctx, st) : nullptr;
        launch_extend(ctx, blocks, st, wide, src, q.ext[buf], ctl, S);
        nan_host::timing_end(ctx, 0, ev, st);
        ctx->launches++;
    }
    if (it > 0u || gen_shadows) {
        cudaEvent_t ev = timed ? nan_host::timing_begin(ctx, st) : nullptr;
        launch_shadow(ctx, blocks, st, wide, src, q.shd[buf ^ 1], ctl - kCtlWords, t_max, S);
        nan_host::timing_end(ctx, 1, ev, st);
        ctx->launches++;
    }
}

}  // namespace

namespace nan_host {

size_t wavefront_bytes_per_path() { return kBytesPerPath + 64; }

namespace {
cudaEvent_t pooled_event(NanContext* ctx) {
    if (!ctx->event_pool.empty()) {
        cudaEvent_t e = ctx->event_pool.back();
        ctx->event_pool.pop_back();
        return e;
    }
    cudaEvent_t e = nullptr;
    if (cudaEventCreate(&e) != cudaSuccess) return nullptr;
    return e;
}
}  // namespace

cudaEvent_t timing_begin(NanContext* ctx, cudaStream_t stream) {
    if (!ctx->tuning.kernel_timing) return nullptr;
    cudaEvent_t e = pooled_event(ctx);
    if (e && cudaEventRecord(e, stream) != cudaSuccess) {
        ctx->event_pool.push_back(e);
        return nullptr;
    }
    return e;
}

void timing_end(NanContext* ctx, int kind, cudaEvent_t start, cudaStream_t stream) {
    if (!start) return;
    cudaEvent_t e = pooled_event(ctx);
    if (!e || cudaEventRecord(e, stream) != cudaSuccess) {
        ctx->event_pool.push_back(start);
        if (e) ctx->event_pool.push_back(e);
        return;
    }
    ctx->timed.push_back({kind, start, e});
}

int read_kernel_times(NanContext* ctx, NanKernelTimes* out, int reset) {
    cudaError_t first = cudaSuccess;
    for (const NanContext::TimedLaunch& t : ctx->timed) {
        float ms = 0.0f;
        cudaError_t err = cudaEventSynchronize(t.stop);
        if (err == cudaSuccess) err = cudaEventElapsedTime(&ms, t.start, t.stop);
        if (err == cudaSuccess) {
            ctx->stage_ms[t.kind] += ms;
            ctx->stage_launches[t.kind]++;
        } else if (first == cudaSuccess) {
            first = err;
        }
        ctx->event_pool.push_back(t.start);
        ctx->event_pool.push_back(t.stop);
    }
    ctx->timed.clear();
    if (out) {
        out->extend_ms = ctx->stage_ms[0];
        out->shadow_ms = ctx->stage_ms[1];
        out->stage_ms = ctx->stage_ms[2];
        out->extend_launches = ctx->stage_launches[0];
        out->shadow_launches = ctx->stage_launches[1];
        out->stage_launches = ctx->stage_launches[2];
    }
    if (reset) {
        for (int k = 0; k < 3; ++k) {
            ctx->stage_ms[k] = 0.0;
            ctx->stage_launches[k] = 0;
        }
    }
    return cuda_fail(first, "kernel timing events");
}

void release_timing(NanContext* ctx) {
    for (const NanContext::TimedLaunch& t : ctx->timed) {
        cudaEventDestroy(t.start);
        cudaEventDestroy(t.stop);
    }
    ctx->timed.clear();
    for (cudaEvent_t e : ctx->event_pool) cudaEventDestroy(e);
    ctx->event_pool.clear();
}

// Scratch plan shared by the integrators: `samples` samples of up to `bounces`
// traced vertices each take bounces + 1 rounds (the last one closes); control
// words for them plus as many paths as the arena holds (or the tuning cap).
// 8 words a round, at most 2 rounds per bounce, fit the 20 words a bounce
// set aside.
int wf_plan(NanContext* ctx, uint64_t samples, uint32_t bounces, uint32_t* rounds, uint64_t* cap) {
    const uint64_t iters64 = samples * bounces;
    if (iters64 > (1u << 20)) {
        set_error("samples * bounces too large for the wavefront schedule");
        return NAN_ERR_INVALID_ARGUMENT;
    }
    *rounds = (uint32_t)(samples * (bounces + 1u));
    const size_t ctl_bytes = ((size_t)(iters64 + 2) * 20 * sizeof(uint32_t) + 255u) / 256u * 256u;
    static_assert(20 >= 2 * kCtlWords, "control words");
    if (ctx->scratch_bytes <= ctl_bytes + 8192) {
        set_error("no wavefront scratch reserved on this context (nan_ctx_reserve)");
        return NAN_ERR_INVALID_ARGUMENT;
    }
    *cap = (ctx->scratch_bytes - ctl_bytes - 8192) / wavefront_bytes_per_path();
    if (ctx->tuning.max_paths_in_flight) *cap = std::min<uint64_t>(*cap, ctx->tuning.max_paths_in_flight);
    if (*cap == 0) {
        set_error("wavefront scratch too small for one path");
        return NAN_ERR_INVALID_ARGUMENT;
    }
    return NAN_OK;
}

size_t ctl_words(uint32_t rounds) { return (size_t)(rounds + 2) * kCtlWords + 16; }

void wf_carve(NanContext* ctx, uint32_t count, uint32_t rounds, WfState& S, WfQueues& q) {
    unsigned char* cur = static_cast<unsigned char*>(ctx->scratch);
    q.ctl = carve<uint32_t>(cur, ctl_words(rounds));
    q.oct = q.ctl + (size_t)(rounds + 2) * kCtlWords;
    q.cap = count;
    S.unit = carve<uint32_t>(cur, count);
    S.rng = carve<uint32_t>(cur, count);
    S.flags = carve<uint32_t>(cur, count);
    S.surf = carve<float4>(cur, count);
    S.ro = carve<float4>(cur, count);
    S.rd = carve<float4>(cur, count);
    S.thp = carve<float4>(cur, count);
    S.rad = carve<float4>(cur, count);
    S.si = carve<float4>(cur, count);
    S.irr = carve<float4>(cur, count);
    S.zpdf = carve<float2>(cur, count);
    S.hit = carve<float4>(cur, count);
    S.pa = carve<float4>(cur, count);
    S.pb = carve<uint4>(cur, count);
    S.pc = carve<uint4>(cur, 2ull * count);
    q.ext[0] = carve<uint32_t>(cur, count);
    q.ext[1] = carve<uint32_t>(cur, count);
    q.ext_sorted = carve<uint32_t>(cur, count);
    q.shd[0] = carve<float4>(cur, 3ull * 2 * count);
    q.shd[1] = carve<float4>(cur, 3ull * 2 * count);
}

// Runs units [begin, end) in chunks: generate, then `rounds` rounds of trace
// and stage. gen(S, q, first_unit, count) and stage(S, q, buf, ctl, blocks)
// launch the integrator's own stages. The control block of round k is block
// k + 1: the generated paths' shadow rays (gen_shadows: there may be some)
// belong to block 0.
template <class Gen, class Stage>
int wf_run(NanContext* ctx, cudaStream_t st, uint64_t begin, uint64_t end, uint32_t rounds, uint64_t cap, float t_max,
           bool gen_shadows, Gen gen, Stage stage) {
    const SceneView s = scene_view(ctx);
    const Grid g = grid_for(ctx, std::min<uint64_t>(cap, end - begin));
    for (uint64_t cb = begin; cb < end; cb += cap) {
        const uint32_t count = (uint32_t)std::min<uint64_t>(cap, end - cb);
        WfState S;
        WfQueues q;
        wf_carve(ctx, count, rounds, S, q);
        cudaError_t err = cudaMemsetAsync(q.ctl, 0, ctl_words(rounds) * sizeof(uint32_t), st);
        if (err != cudaSuccess) return cuda_fail(err, "wavefront control reset");
        cudaEvent_t ev = timing_begin(ctx, st);
        gen(S, q, (uint32_t)cb, count);
        timing_end(ctx, 2, ev, st);
        ctx->launches++;
        for (uint32_t it = 0; it < rounds; ++it) {
            const int buf = (int)(it & 1u);
            uint32_t* ctl = q.ctl + kCtlWords * (it + 1u);
            if (ctx->tuning.ray_order == 1u) {
                ev = timing_begin(ctx, st);
                err = cudaMemsetAsync(q.oct, 0, 16 * sizeof(uint32_t), st);
                if (err != cudaSuccess) return cuda_fail(err, "ray order reset");
                k_wf_octant_count<<<g.stream_blocks, 256, 0, st>>>(q.ext[buf], ctl, S.rd, q.oct);
                k_wf_octant_place<<<g.stream_blocks, 256, 0, st>>>(q.ext[buf], ctl, S.rd, q.oct, q.ext_sorted);
                k_wf_close_copy<<<g.stream_blocks, 256, 0, st>>>(q.ext[buf], ctl, q.cap, q.ext_sorted);
                timing_end(ctx, 2, ev, st);
                std::swap(q.ext[buf], q.ext_sorted);
                ctx->launches += 3;
            }
            launch_trace(ctx, g.persistent_blocks, st, s.wnodes != nullptr, true, gen_shadows, OneScene{s}, q, it, rounds, t_max, S);
            ev = timing_begin(ctx, st);
            stage(S, q, buf, ctl, g.stream_blocks);
            timing_end(ctx, 2, ev, st);
            ctx->launches++;
        }
        err = cudaGetLastError();
        if (err != cudaSuccess) return cuda_fail(err, "wavefront launch");
    }
    return NAN_OK;
}

int launch_trace_texels_wavefront(NanContext* ctx, const NanMeshColorsDesc* lay, uint8_t* slots,
                                  uint32_t iteration, uint32_t spt, uint32_t max_bounces, int reset,
                                  const NanLighting* light, uint32_t begin, uint32_t end, cudaStream_t st) {
    if (end <= begin) return NAN_OK;
    const uint32_t n = std::max(spt, 1u);
    uint32_t rounds = 0;
    uint64_t cap = 0;
    // a path may run its back side after its front: 2 sides x n samples
    int rc = wf_plan(ctx, 2ull * n, std::max(max_bounces, 1u), &rounds, &cap);
    if (rc) return rc;
    const SceneView s = scene_view(ctx);
    const LightingRaw lr = to_raw(light);
    TexelArgs a;
    memset(&a, 0, sizeof(a));
    a.mc.compensation = reinterpret_cast<float4*>(lay->compensation);
    a.mc.face_infos = reinterpret_cast<const uint2*>(lay->face_infos);
    a.mc.instance_infos = reinterpret_cast<const uint4*>(lay->instance_infos);
    a.mc.side_infos = reinterpret_cast<const uint2*>(lay->side_infos);
    a.mc.surface_prefix = lay->surface_prefix;
    a.mc.instance_count = lay->instance_count;
    a.mc.payload_count = lay->payload_count;
    a.slots = reinterpret_cast<uint4*>(slots);
    a.iteration = iteration;
    a.n = n;
    a.max_bounces = std::max(max_bounces, 1u);
    a.reset = reset;
    unsigned long long* counters = ctx->d_counters;
    return wf_run(
        ctx, st, begin, end, rounds, cap, lr.ray_t_max, true,
        [&](const WfState& S, const WfQueues& q, uint32_t first, uint32_t count) {
            k_wf_texel_generate<<<(count + kStageThreads - 1) / kStageThreads, kStageThreads, 0, st>>>(s, lr, a, S, q, first, count, counters);
        },
        [&](const WfState& S, const WfQueues& q, int buf, uint32_t* ctl, int blocks) {
            k_wf_texel_stage<<<blocks, kStageThreads, 0, st>>>(s, lr, a, S, q, buf, ctl);
        });
}

namespace {
int screen_wavefront(NanContext* ctx, float* out, uint32_t w, uint32_t h, uint32_t frame, uint32_t max_vertices,
                     const NanCamera* cam, const NanLighting* light, const CachedArgs* cached, cudaStream_t st);
}  // namespace

int launch_trace_screen_wavefront(NanContext* ctx, float* out, uint32_t w, uint32_t h, uint32_t frame,
                                  uint32_t max_vertices, const NanCamera* cam, const NanLighting* light,
                                  cudaStream_t st) {
    return screen_wavefront(ctx, out, w, h, frame, max_vertices, cam, light, nullptr, st);
}

int launch_trace_screen_cached(NanContext* ctx, NanCache* cache, float* out, uint32_t w, uint32_t h,
                               uint32_t frame, const NanCamera* cam, const NanLighting* light,
                               const NanCachedFrame* fd, cudaStream_t st) {
    CachedArgs c;
    c.queries = reinterpret_cast<float4*>(fd->queries);
    c.weights = reinterpret_cast<float4*>(fd->query_weights);
    c.query_count = fd->query_count;
    c.train_points = reinterpret_cast<float4*>(fd->train_points);
    c.train_queries = reinterpret_cast<float4*>(fd->train_queries);
    c.train_count = fd->train_count;
    c.train_offset = fd->train_offset;
    c.train_inverse = fd->train_stride_inverse;
    c.vertex = fd->cache_vertex;
    cudaError_t err = cudaMemsetAsync(fd->query_count, 0, sizeof(uint32_t), st);
    if (err == cudaSuccess && fd->train_count)
        err = cudaMemsetAsync(fd->train_points, 0xff, (size_t)fd->train_count * 16u, st);
    if (err != cudaSuccess) return cuda_fail(err, "cached frame reset");
    int rc = screen_wavefront(ctx, out, w, h, frame, fd->cache_vertex + 1u, cam, light, &c, st);
    if (rc) return rc;
    return launch_cache_infer(cache, fd->queries, w * h, fd->query_count, nullptr, fd->query_weights, out, st);
}

int launch_trace_points_wavefront(NanContext* ctx, const float* points, uint32_t count, float* out,
                                  uint32_t iteration, uint32_t samples, uint32_t max_bounces, uint32_t flags,
                                  const NanLighting* light, cudaStream_t st) {
    if (count == 0) return NAN_OK;
    const uint32_t n = std::max(samples, 1u);
    uint32_t rounds = 0;
    uint64_t cap = 0;
    int rc = wf_plan(ctx, n, std::max(max_bounces, 1u), &rounds, &cap);
    if (rc) return rc;
    const SceneView s = scene_view(ctx);
    const LightingRaw lr = to_raw(light);
    TexelArgs a;
    memset(&a, 0, sizeof(a));
    a.iteration = iteration;
    a.n = n;
    a.max_bounces = std::max(max_bounces, 1u);
    a.points = reinterpret_cast<const float4*>(points);
    a.point_out = reinterpret_cast<float4*>(out);
    a.indirect_only = (flags & NAN_POINTS_INDIRECT_ONLY) != 0u;
    unsigned long long* counters = ctx->d_counters;
    return wf_run(
        ctx, st, 0, count, rounds, cap, lr.ray_t_max, !a.indirect_only,
        [&](const WfState& S, const WfQueues& q, uint32_t first, uint32_t cnt) {
            k_wf_point_generate<<<(cnt + kStageThreads - 1) / kStageThreads, kStageThreads, 0, st>>>(s, lr, a, S, q, first, cnt, counters);
        },
        [&](const WfState& S, const WfQueues& q, int buf, uint32_t* ctl, int blocks) {
            k_wf_texel_stage<<<blocks, kStageThreads, 0, st>>>(s, lr, a, S, q, buf, ctl);
        });
}

namespace {
int screen_wavefront(NanContext* ctx, float* out, uint32_t w, uint32_t h, uint32_t frame, uint32_t max_vertices,
                     const NanCamera* cam, const NanLighting* light, const CachedArgs* cached, cudaStream_t st) {
    const uint64_t pixels = (uint64_t)w * h;
    if (pixels == 0 || max_vertices == 0) return NAN_OK;
    uint32_t rounds = 0;
    uint64_t cap = 0;
    int rc = wf_plan(ctx, 1u, max_vertices, &rounds, &cap);
    if (rc) return rc;
    const SceneView s = scene_view(ctx);
    const LightingRaw lr = to_raw(light);
    ScreenArgs a;
    memcpy(&a.cam, cam, sizeof(a.cam));
    a.out = reinterpret_cast<float4*>(out);
    a.width = w;
    a.height = h;
    a.frame = frame;
    a.max_vertices = max_vertices;
    a.cached = cached != nullptr;
    if (cached) a.cache = *cached;
    else memset(&a.cache, 0, sizeof(a.cache));
    unsigned long long* counters = ctx->d_counters;
    return wf_run(
        ctx, st, 0, pixels, rounds, cap, lr.ray_t_max, false,
        [&](const WfState& S, const WfQueues& q, uint32_t first, uint32_t count) {
            k_wf_screen_generate<<<(count + kStageThreads - 1) / kStageThreads, kStageThreads, 0, st>>>(s, lr, a, S, q, first, count, counters);
        },
        [&](const WfState& S, const WfQueues& q, int buf, uint32_t* ctl, int blocks) {
            k_wf_screen_stage<<<blocks, kStageThreads, 0, st>>>(s, lr, a, S, q, buf, ctl);
        });
}
}  // namespace

size_t probe_sample_bytes() { return sizeof(ProbeSample); }

const void* wavefront_extend_kernel() { return reinterpret_cast<const void*>(&k_wf_trace<2, ManyScenes>); }

// The multi-scene probe batch on the wavefront: generate every (set, probe)
// unit as one path, then n * (max_bounces + 1) rounds of a trace and a stage
// launch over all sets, with no host synchronisation (capturable). The
// context's scratch must hold `total` paths.
int launch_batch_wavefront(NanContext* ctx, const void* sets, const uint32_t* prefix, const void* batch_ctl,
                           uint32_t set_count, uint32_t total, uint32_t* set_of, uint32_t spp, uint32_t max_bounces,
                           float t_max, cudaStream_t st) {
    if (total == 0) return NAN_OK;
    const uint32_t n = std::max(spp, 1u);
    uint32_t rounds = 0;
    uint64_t cap = 0;
    int rc = wf_plan(ctx, n, std::max(max_bounces, 1u), &rounds, &cap);
    if (rc) return rc;
    if (cap < total) {
        set_error("batch wavefront scratch holds fewer paths than the batch has probes");
        return NAN_ERR_INVALID_ARGUMENT;
    }
    BatchWfArgs m;
    m.sets = static_cast<const BatchSet*>(sets);
    m.prefix = prefix;
    m.ctl = static_cast<const BatchCtl*>(batch_ctl);
    m.set_of = set_of;
    m.set_count = set_count;
    m.total = total;
    m.n = n;
    m.spp = spp;
    m.max_bounces = std::max(max_bounces, 1u);
    m.unit_begin = 0u;
    m.units = total;
    m.samples = nullptr;
    const ManyScenes src{m.sets, set_of};
    const Grid g = grid_for(ctx, total);
    WfState S;
    WfQueues q;
    wf_carve(ctx, total, rounds, S, q);
    cudaError_t err = cudaMemsetAsync(q.ctl, 0, ctl_words(rounds) * sizeof(uint32_t), st);
    if (err != cudaSuccess) return cuda_fail(err, "batch wavefront control reset");
    k_wfb_probe_generate<<<(total + kStageThreads - 1) / kStageThreads, kStageThreads, 0, st>>>(m, S, q, ctx->d_counters);
    ctx->launches++;
    for (uint32_t it = 0; it < rounds; ++it) {
        launch_trace(ctx, g.persistent_blocks, st, false, false, false, src, q, it, rounds, t_max, S);
        k_wfb_probe_stage<<<g.stream_blocks, kStageThreads, 0, st>>>(m, S, q, (int)(it & 1u), q.ctl + kCtlWords * (it + 1u));
        ctx->launches++;
    }
    return cuda_fail(cudaGetLastError(), "batch wavefront launch");
}

int launch_batch_wavefront_independent(NanContext* ctx, const void* sets, const uint32_t* prefix,
                                       const void* batch_ctl, uint32_t set_count, uint32_t total, uint32_t* set_of,
                                       void* samples, uint64_t path_capacity, uint32_t spp, uint32_t max_bounces,
                                       float t_max, cudaStream_t st) {
    if (total == 0) return NAN_OK;
    const uint32_t n = std::max(spp, 1u);
    uint32_t rounds = 0;
    uint64_t cap = 0;
    int rc = wf_plan(ctx, 1u, std::max(max_bounces, 1u), &rounds, &cap);
    if (rc) return rc;
    cap = std::min(cap, path_capacity);
    const uint64_t chunk_units = cap / n;
    if (chunk_units == 0) {
        set_error("batch wavefront scratch holds fewer paths than one probe's samples");
        return NAN_ERR_INVALID_ARGUMENT;
    }
    BatchWfArgs m;
    m.sets = static_cast<const BatchSet*>(sets);
    m.prefix = prefix;
    m.ctl = static_cast<const BatchCtl*>(batch_ctl);
    m.set_of = set_of;
    m.set_count = set_count;
    m.total = total;
    m.n = n;
    m.spp = spp;
    m.max_bounces = std::max(max_bounces, 1u);
    m.samples = static_cast<ProbeSample*>(samples);
    const ManyScenes src{m.sets, set_of};
    const Grid g = grid_for(ctx, std::min<uint64_t>(chunk_units, total) * n);
    for (uint64_t ub = 0; ub < total; ub += chunk_units) {
        m.unit_begin = (uint32_t)ub;
        m.units = (uint32_t)std::min<uint64_t>(chunk_units, total - ub);
        const uint32_t paths = m.units * n;
        WfState S;
        WfQueues q;
        wf_carve(ctx, paths, rounds, S, q);
        cudaError_t err = cudaMemsetAsync(q.ctl, 0, ctl_words(rounds) * sizeof(uint32_t), st);
        if (err != cudaSuccess) return cuda_fail(err, "batch wavefront control reset");
        k_wfi_probe_generate<<<(paths + kStageThreads - 1) / kStageThreads, kStageThreads, 0, st>>>(m, S, q);
        for (uint32_t it = 0; it < rounds; ++it) {
            launch_trace(ctx, g.persistent_blocks, st, false, false, false, src, q, it, rounds, t_max, S);
            k_wfi_probe_stage<<<g.stream_blocks, kStageThreads, 0, st>>>(m, S, q, (int)(it & 1u), q.ctl + kCtlWords * (it + 1u));
        }
        k_wfi_probe_fold<<<(m.units + 127) / 128, 128, 0, st>>>(m, ctx->d_counters);
        ctx->launches += 2 + rounds;
    }
    return cuda_fail(cudaGetLastError(), "batch wavefront launch");
}

int launch_trace_probes_wavefront(NanContext* ctx, float* values, uint32_t* counts, uint32_t* self_hits,
                                  uint32_t* radial, const uint8_t* probes, uint32_t probe_count,
                                  const uint8_t* probe_instances, uint32_t probe_instance_count, uint32_t iteration,
                                  uint32_t spp, uint32_t max_bounces, int reset, const NanLighting* light,
                                  uint32_t begin, uint32_t end, float* compensation, cudaStream_t st) {
    end = std::min(end, probe_count);
    if (end <= begin) return NAN_OK;
    const uint32_t n = std::max(spp, 1u);
    uint32_t rounds = 0;
    uint64_t cap = 0;
    int rc = wf_plan(ctx, n, std::max(max_bounces, 1u), &rounds, &cap);
    if (rc) return rc;
    const SceneView s = scene_view(ctx);
    const LightingRaw lr = to_raw(light);
    ProbeArgs a;
    a.out = ProbeOut{reinterpret_cast<float4*>(compensation), values, counts, self_hits, radial};
    a.probes = reinterpret_cast<const float4*>(probes);
    a.pinst = reinterpret_cast<const float4*>(probe_instances);
    a.probe_instance_count = probe_instance_count;
    a.iteration = iteration;
    a.n = n;
    a.spp = spp;
    a.max_bounces = std::max(max_bounces, 1u);
    a.reset = reset;
    unsigned long long* counters = ctx->d_counters;
    return wf_run(
        ctx, st, begin, end, rounds, cap, lr.ray_t_max, false,
        [&](const WfState& S, const WfQueues& q, uint32_t first, uint32_t count) {
            k_wf_probe_generate<<<(count + kStageThreads - 1) / kStageThreads, kStageThreads, 0, st>>>(s, lr, a, S, q, first, count, counters);
        },
        [&](const WfState& S, const WfQueues& q, int buf, uint32_t* ctl, int blocks) {
            k_wf_probe_stage<<<blocks, kStageThreads, 0, st>>>(s, lr, a, S, q, buf, ctl);
        });
}

}  // namespace nan_host
