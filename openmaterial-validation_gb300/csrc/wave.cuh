// Building blocks of the wavefront pipelines (the renderer's and the
// path-replay adjoint's): queue appends, division by frame constants, the
// light pick, the closest-hit loop over a ray queue and the connection test.
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "omv_device.cuh"
#include "shade.cuh"
#include "trace.cuh"

namespace omv {

constexpr int kTraceThreads = 128;
// 6 resident blocks of the trace kernels per SM (80 registers, a few spilled
// stack words): more warps in flight for the latency-bound traversal than the
// 5 blocks its unconstrained 96 registers allow (measured 3.18 -> 3.06 ms per
// extension launch on the 1920x1080x64 frame; 7 and 8 blocks spill more)
constexpr int kTraceMinBlocks = 6;
constexpr int kShadeThreads = 256;

__device__ __forceinline__ uint32_t warp_append(uint32_t* counter, bool want)
{
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, want);
    if (!m) return 0;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(m) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(counter, (uint32_t)__popc(m));
    base = __shfl_sync(0xFFFFFFFFu, base, leader);
    return base + __popc(m & ((1u << lane) - 1u));
}

// Opportunistic warp aggregation (for appends inside divergent code): the
// threads of a warp that arrive together take consecutive slots with one atomic.
__device__ __forceinline__ uint32_t coalesced_append(uint32_t* counter)
{
    namespace cg = cooperative_groups;
    const cg::coalesced_group g = cg::coalesced_threads();
    uint32_t base = 0;
    if (g.thread_rank() == 0) base = atomicAdd(counter, (uint32_t)g.size());
    return g.shfl(base, 0) + (uint32_t)g.thread_rank();
}

// Direction bin of a ray: the cube face its direction points to (dominant
// axis and sign) and the quadrant on that face, 24 bins.
constexpr int kDirBins = 24;
__device__ __forceinline__ uint32_t direction_bin(V3 d)
{
    const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    uint32_t f;
    float u, v;
    if (ax >= ay && ax >= az) {
        f = d.x < 0.0f ? 1u : 0u;
        u = d.y;
        v = d.z;
    } else if (ay >= az) {
        f = d.y < 0.0f ? 3u : 2u;
        u = d.z;
        v = d.x;
    } else {
        f = d.z < 0.0f ? 5u : 4u;
        u = d.x;
        v = d.y;
    }
    return 4u * f + (u < 0.0f ? 2u : 0u) + (v < 0.0f ? 1u : 0u);
}

struct BinScratch {
    uint32_t count[kDirBins];
    uint32_t base;
};

// Block-wide append to a queue with the block's entries grouped by bin, so
// that the warps tracing the queue get rays of similar direction from nearby
// pixels.  One atomic per block; every thread of the block must call it.
__device__ __forceinline__ uint32_t block_append_binned(uint32_t* counter, bool want, uint32_t bin, BinScratch& sh)
{
    if (threadIdx.x < kDirBins) sh.count[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t rank = want ? atomicAdd(&sh.count[bin], 1u) : 0u;
    __syncthreads();
    if (threadIdx.x < 32) {
        // exclusive scan of the bin counts in the first warp; lane 31 reserves
        const uint32_t c = threadIdx.x < kDirBins ? sh.count[threadIdx.x] : 0u;
        uint32_t x = c;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if ((int)threadIdx.x >= o) x += y;
        }
        if (threadIdx.x < kDirBins) sh.count[threadIdx.x] = x - c;
        if (threadIdx.x == 31) sh.base = x ? atomicAdd(counter, x) : 0u;
    }
    __syncthreads();
    const uint32_t slot = sh.base + sh.count[bin] + rank;
    __syncthreads();  // the scratch is reused by the next call
    return slot;
}

// The next rays of a block's window of kStageSteps steps, kept in shared memory
// and then appended to the queue grouped by direction: four times the rays of
// block_append_binned per group, and its barriers once per window instead of
// once per step (32 KB per block; kStagedPaths says where it pays).
constexpr int kStageSteps = 4;
constexpr uint32_t kStageWindows = 8;
struct StagedRays {
    float4 ray[2 * kStageSteps * kShadeThreads];
    uint32_t count[32];  // per bin, then the bin's start
    uint32_t n, base;
};
// every thread of the block calls the three; staged_add by whole warps
__device__ __forceinline__ void staged_begin(StagedRays& s)
{
    if (threadIdx.x < 32) s.count[threadIdx.x] = 0;
    if (threadIdx.x == 0) s.n = 0;
    __syncthreads();
}
__device__ __forceinline__ void staged_add(StagedRays& s, bool want, float4 a, float4 b)
{
    const uint32_t at = warp_append(&s.n, want);
    if (want) {
        s.ray[2 * at] = a;
        s.ray[2 * at + 1] = b;
    }
}
__device__ __forceinline__ void staged_append(StagedRays& s, uint32_t* counter, float4* queue)
{
    __syncthreads();
    const uint32_t n = s.n;
    uint32_t bin[kStageSteps], rank[kStageSteps];
#pragma unroll
    for (int j = 0; j < kStageSteps; ++j) {
        const uint32_t t = j * blockDim.x + threadIdx.x;
        if (t < n) {
            const float4 d = s.ray[2 * t + 1];
            bin[j] = direction_bin(v3(d.x, d.y, d.z));
            rank[j] = atomicAdd(&s.count[bin[j]], 1u);
        }
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const uint32_t c = s.count[threadIdx.x];
        uint32_t x = c;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if ((int)threadIdx.x >= o) x += y;
        }
        s.count[threadIdx.x] = x - c;
        if (threadIdx.x == 31) s.base = x ? atomicAdd(counter, x) : 0u;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kStageSteps; ++j) {
        const uint32_t t = j * blockDim.x + threadIdx.x;
        if (t < n) {
            float4* q = queue + 2 * ((size_t)s.base + s.count[bin[j]] + rank[j]);
            q[0] = s.ray[2 * t];
            q[1] = s.ray[2 * t + 1];
        }
    }
    __syncthreads();  // the window's rays are read before the next one's come
}

// Division of 32-bit unsigned integers by a divisor fixed for a frame, by one
// multiply-high, a subtraction and two shifts (Granlund & Montgomery,
// "Division by invariant integers using multiplication", PLDI 1994, 4.1):
// exact for every numerator and every divisor >= 1, where the hardware has
// no integer divide.
inline FastDiv make_fastdiv(uint32_t d)
{
    int l = 0;
    while (l < 32 && (1ull << l) < d) ++l;
    FastDiv f;
    f.d = d;
    f.m = (uint32_t)(((((1ull << l) - d) << 32) / d) + 1);
    f.s1 = l < 1 ? l : 1;
    f.s2 = l > 1 ? l - 1 : 0;
    return f;
}
__device__ __forceinline__ uint32_t fast_div(const FastDiv& f, uint32_t n)
{
    const uint32_t t1 = __umulhi(f.m, n);
    return (t1 + ((n - t1) >> f.s1)) >> f.s2;
}

// DistanceRandom::getValue (DistanceRandom.h:98-115): the light of a draw d
// from the power CDF of n > 1 lights
__device__ __forceinline__ int pick_light(const float* cdf, int n, float d)
{
    if (d <= cdf[0]) return 0;
    if (d >= cdf[n - 2]) return n - 1;
    int L = 0, R = n - 1;
    while (L < R) {
        const int C = (L + R) / 2;
        if (d <= cdf[C])
            R = C;
        else
            L = C + 1;
    }
    return (L + R) / 2;
}

// The rays of a persistent tracing launch, in shares that its warps draw from
// an atomic counter: kBigShare steps of `take` rays while many are left, single
// steps for the last kSmallRays (large shares there leave some warps with much
// more work than others: from 2^22 on, an 8.4M-ray launch 0.53 -> 0.71 ms).  The
// counter is one address, which takes about one atomic per nanosecond: a draw
// per 32 rays bounds a launch at 24 G rays/s, and the first bounce of the
// 1920x1080x64 sky frame took 5.5 ms from its tile lists with it, 2.3 so.
// Warp w starts with share w, so a launch with at most a share per warp makes
// no atomic at all (empty: 5.1 -> 2.8 us).
constexpr uint32_t kBigShare = 8, kSmallRays = 1u << 23;
// Only the next ray's number lives across a step: a share of several steps ends
// at a multiple of its size.
struct RayShares {
    uint32_t next;
};
__device__ __forceinline__ uint32_t share_start(uint32_t j, uint32_t take, uint32_t n)
{
    const uint32_t span = kBigShare * take, big = n > kSmallRays ? (n - kSmallRays) / span : 0u;
    if (j < big) return j * span;
    const uint64_t at = (uint64_t)big * span + (uint64_t)(j - big) * take;
    return at < n ? (uint32_t)at : 0xFFFFFFFFu;
}
__device__ __forceinline__ RayShares ray_shares(uint32_t take, uint32_t n)
{
    return RayShares{share_start(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), take, n)};
}
// after a step: the warp's next one
__device__ __forceinline__ void next_step(RayShares& s, uint32_t take, uint32_t n, uint32_t* work)
{
    const uint32_t span = kBigShare * take, at = s.next + take;
    const uint32_t big_end = n > kSmallRays ? (n - kSmallRays) / span * span : 0u;
    if (at <= big_end && at % span != 0u) {
        s.next = at;
        return;
    }
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    if (big_end == 0u && (uint64_t)warps * take >= n) {  // all shares were first shares
        s.next = 0xFFFFFFFFu;
        return;
    }
    uint32_t x = 0;
    if ((threadIdx.x & 31) == 0) x = atomicAdd(work, 1u);
    s.next = share_start(warps + __shfl_sync(0xFFFFFFFFu, x, 0), take, n);
}

// Queues of at most this many rays are traced with eight lanes per ray
// (coop_trace), longer ones with one ray per thread: a 256x256x16 point-light
// frame 947 us with the line at 2^15 (952 at 2^14, 959 at 2^16, 1013 at 2^17),
// an eight-scene inverse-fit step 5.26 ms (5.25, 5.28, 5.51).  What the path
// gave when it was added, before the second stream: the same frame 1245 -> 1121
// us, a 64x64x1 one 728 -> 532, the step 5.99 -> 5.78 ms.
constexpr uint32_t kCoopRays = 1u << 15;
static_assert(kStackShared * kTraceThreads >= kStackTotal * (kTraceThreads / kCoopLanes),
              "the groups of a block share its stacks' memory");

// The eight-lane groups of a warp and their part of the block's stack memory.
struct CoopGroup {
    uint32_t mask;
    int sub, index;  // lane in the group, group in the warp
    CoopStack st;
};
__device__ __forceinline__ CoopGroup coop_group(uint2* stacks)
{
    CoopGroup g;
    const int lane = threadIdx.x & 31;
    g.sub = lane & (kCoopLanes - 1);
    g.index = lane / kCoopLanes;
    g.mask = ((1u << kCoopLanes) - 1u) << (g.index * kCoopLanes);
    g.st.sh = stacks + (threadIdx.x / kCoopLanes) * kStackTotal;
    g.st.sp = 0;
    g.st.overflow = 0;
    return g;
}

// Persistent closest hit over the n rays of a queue: a warp takes 32 consecutive rays and the next 32 when all are done
// (camera rays: the 32 samples of one pixel stay together).  Replacing
// finished rays lane by lane (Aila & Laine 2009) was measured slower on every
// bounce.  root(k): the top-level tree of path k's scene (k travels in the
// ray's last word).  Short queues: four rays per warp.
template <typename Root>
__device__ __forceinline__ void extend_rays(const DevScene& S, const uint32_t* items, float4* rq, uint4* hits,
                                            uint32_t n, uint32_t* work, TraceStack& st, TraceCounters& tc, Root root)
{
    const int lane = threadIdx.x & 31;
    for (RayShares s = ray_shares(32u, n); s.next < n; next_step(s, 32u, n, work)) {
        const uint32_t base = s.next;
        const uint32_t i = base + lane;
        if (i < n) {
            float4 a = rq[2 * (size_t)i], b = rq[2 * (size_t)i + 1];
            V3 o = v3(a.x, a.y, a.z), d = v3(b.x, b.y, b.z);
            float tnear = a.w;
            RayHit h;
            uint4 out;
            if (scene_intersect(S, items, o, d, tnear, kFltMax, h, st, tc, root(__float_as_int(b.w))))
                out = make_uint4(h.inst, h.prim, __float_as_uint(h.u), __float_as_uint(h.v));
            else
                out = make_uint4(kInvalid, kInvalid, 0u, 0u);
            hits[i] = out;
            if (tnear != a.w) rq[2 * (size_t)i].w = tnear;
        }
    }
}

// what a call on the eight-lane path counted
struct CoopCounts {
    TraceCounters tc;
    int overflow;
};

// extend_rays for short queues, four rays per warp.  Out of line, so that its
// registers do not weigh on the one-thread path of the same kernel.
template <typename Root>
__device__ __noinline__ CoopCounts extend_rays_coop(const DevScene& S, const uint32_t* items, float4* rq, uint4* hits,
                                                    uint32_t n, uint32_t* work, uint2* stacks, Root root)
{
    CoopGroup g = coop_group(stacks);
    TraceCounters tc{0u, 0u};
    for (RayShares s = ray_shares(32u / kCoopLanes, n); s.next < n; next_step(s, 32u / kCoopLanes, n, work)) {
        const uint32_t base = s.next;
        const uint32_t i = base + (uint32_t)g.index;
        if (i < n) {
            const float4 a = rq[2 * (size_t)i], b = rq[2 * (size_t)i + 1];
            float tnear = a.w;
            RayHit h;
            const bool hit = coop_intersect(S, items, v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), tnear, kFltMax, h, g.st, tc,
                                            root(__float_as_int(b.w)), g.mask, g.sub);
            if (g.sub == 0) {
                hits[i] = hit ? make_uint4(h.inst, h.prim, __float_as_uint(h.u), __float_as_uint(h.v))
                              : make_uint4(kInvalid, kInvalid, 0u, 0u);
                if (tnear != a.w) rq[2 * (size_t)i].w = tnear;
            }
        }
        __syncwarp();
    }
    return CoopCounts{tc, g.st.overflow};
}

// BDPTRenderer::isConnected (BDPTRenderer.cpp:208-235): whether vertex A sees
// vertex B.  Without alpha-masked materials the closest-hit query stops at a
// hit well short of B, which already decides "not connected".  With a group
// `g`, its eight lanes test one connection together.
template <bool kMasked>
__device__ __forceinline__ bool is_connected(const DevScene& S, const uint32_t* items, V3 A, V3 B, TraceStack& st,
                                             TraceCounters& tc, uint32_t root, CoopGroup* g = nullptr)
{
    bool connected = true;
    V3 dir = B - A;
    const float len = sqrtf(dot(dir, dir));
    float maxsz = max_abs(A, 1.0f);
    float safeD = 2.0f * kEpsAcc * kEps * maxsz;
    if (!(len <= safeD)) {
        dir = v3(dir.x / len, dir.y / len, dir.z / len);
        float tnear = safeD;
        const float tfar = len + (0.1f * len > safeD ? 0.1f * len : safeD);
        const float sb = 10.0f * kEps * max_abs(B, 1.0f);
        RayHit h;
        bool hit;
        if (kMasked) {
            hit = g ? coop_intersect(S, items, A, dir, tnear, tfar, h, g->st, tc, root, g->mask, g->sub)
                    : scene_intersect(S, items, A, dir, tnear, tfar, h, st, tc, root);
        } else {
            // any hit this far short of B is farther than sb from it (the
            // margin is ~800 ulps of the coordinates, far above the error of
            // the hit's surface position), so it decides: not connected,
            // whichever hit is the closest.  Hits near B get the exact test.
            const float margin = 1.0e-4f * fmaxf(maxsz, max_abs(B, 1.0f)) + 2.0f * sb;
            hit = g ? coop_trace<true>(S, items, A, dir, tnear, tfar, len - margin, h, g->st, tc, root, g->mask, g->sub)
                    : trace_closest_or_below(S, items, A, dir, tnear, tfar, len - margin, h, st, tc, root);
            if (hit && h.t < len - margin) {
                hit = false;
                connected = false;
            }
        }
        if (hit) {
            const Surf sp = surface_point(S, h.inst, h.prim, h.u, h.v, false);
            const V3 dd = sp.pos - B;
            const float sd = dot(dd, dd);
            connected = sd <= sb * sb;
        }
    }
    return connected;
}

}  // namespace omv
