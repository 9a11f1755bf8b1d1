// Path-replay adjoint of the BDPT estimator (after Vicini, Speierer, Jakob,
// "Path replay backpropagation", SIGGRAPH 2021): gradients of an image loss
// with respect to the material parameters, given the loss's derivative with
// respect to every pixel (the adjoint image).
//
// The replay regenerates every path's light and camera subpath from its Philox
// keys (the same random numbers as the forward render) as a wavefront like the
// renderer's, keeping each vertex's record (ray, hit, throughput, weight), and
// then walks the records backwards, one launch per bounce.  The path's
// estimate is a sum of products of per-vertex factors (BDPTRenderer.cpp:
// 128-302 with weight 1); its derivative is taken with every sampled direction
// held fixed, which for the GGX-sampled branches adds the score d log D / d
// alpha of the half-vector density, so the result is an unbiased estimate of
// the gradient of the expected image (luminance cutoffs are treated as fixed).
// Two division-free backward recursions over the vertices give the factors'
// adjoints:
//   camera  R_b = G_b + w_b R_{b+1}          (k_adj_camera_back)
//   light   S_j = q_j + w_{j+1} S_{j+1}      (k_adj_light_back)
// with G_b the vertex's visible connections and escape term, and q_j the
// adjoint of light vertex j's radiance, both summed by k_adj_connect.
//
// Why a wavefront: the replay was one thread per path with all its vertices and
// their derivatives in local memory (about 7 KB per thread); its warps waited
// for their slowest path, traversal and derivative arithmetic shared 128
// registers, and the records ran through L1 and L2 as local memory.  Split by
// bounce, the traversal kernels are the renderer's, every launch's lanes do the
// same work, and the derivatives, recomputed where the backward walk needs
// them, never leave registers.  One gradient (forward and replay) of 512x512,
// 32 spp, 100k triangles, 8 materials: 111 ms before, 13.1 ms so.  Jobs of a
// batch share the waves: one step of an inverse fit of eight 128x128x16 scenes
// 29 -> 5.26 ms.
//
// Gradients: the lanes of a warp that meet the same material reduce by
// shuffles into the warp's sums in shared memory, the block adds its totals to
// FP64 accumulators, and one last launch adds those to the caller's buffers.
// The total is more exact than a thread's FP32 sums were (error against the sum
// of 64 row bands 2.4e-8, 3.1e-7 before), but not the same from run to run: the
// connections of a vertex are added to its G and to the light vertices' q with
// FP32 atomics in the order in which they come, and the blocks' totals too.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

#include "dual.cuh"
#include "scene.h"
#include "shade.cuh"
#include "wave.cuh"

namespace omv {
namespace {

constexpr int kAdjThreads = 128;
constexpr int kAdjMaxVerts = 16;      // per subpath
constexpr int kAdjMaxMaterials = 16;  // materials with parameters, per scene
constexpr int kSlots = OMV_MATERIAL_PARAMS;
// gradient sums of one wave (jobs x materials x slots): each warp of a block
// keeps all of them in shared memory, 4 x 4 KB
constexpr int kAdjMaxKeys = 1024;

// Counter slots of a wave (reset per wave): queue sizes per bounce, then the
// work counters of the tracing launches.
constexpr int kAdjCtrLight = 0, kAdjCtrCam = 16, kAdjCtrConn = 32, kAdjCtrSeen = 48, kAdjCtrWork = 64,
              kAdjCounters = 128;

// One job of a wave: a scene of the handle, its camera, samples and materials,
// the adjoint image and the gradient buffer.
struct AdjJob {
    omv_camera cam;
    int64_t path_base;  // first path of the wave loop's concatenated paths
    uint64_t seed;
    const DevMaterial* mats;
    const float* adj;   // W*H*3 adjoint image
    float* grad;        // nmat * kSlots
    FastDiv spp_div, width_div;
    int32_t spp, sample_offset;
    uint32_t tlas_root;
    int32_t light_base, light_count;
    float light_max;
    uint32_t mat_base;  // first material of the scene (a scene of a group)
    int32_t nmat;
    int32_t key_base;   // first gradient sum
    float inv_spp;
};
// a table's part that travels as a kernel parameter (a caller may capture the
// call into a graph, where a copy from host memory would be read at replay)
constexpr int kJobsPerPut = 12;
struct AdjJobChunk {
    AdjJob j[kJobsPerPut];
};
static_assert(sizeof(AdjJobChunk) <= 3800, "kernel parameters hold 4 KB");

constexpr int kLenShift = 27;  // lmeta: 15 light vertices at most, 2^27 lights
constexpr uint32_t kLightMask = (1u << kLenShift) - 1u;

// Records of one wave of `cap` paths.  Camera records are kept in queue order
// per bounce, light records by path.
struct AdjWave {
    DevScene S;
    const uint32_t* items;
    const AdjJob* jobs;
    int32_t num_jobs, cap, wave_n, keys;
    int64_t wave_base;
    int32_t cam_bounces, light_bounces, max_len, atten_mode;
    float light_scale, min_dist, cut;
    uint32_t* ctr;
    double* acc;         // gradient sums [keys]
    uint32_t* path_job;  // job of each path (null for one job)
    float4* suffix;      // R of the camera vertices processed so far
    uint32_t* lmeta;     // light index | (light vertices on surfaces << kLenShift)
    float4* ltp;         // light throughput, distance term
    float4* lsuffix;     // w_{j+1} S_{j+1}
    float4 *crq, *ctp, *cw, *cG;  // [bounce][cap]; crq: 2 per entry; ctp.w: the path went on
    uint4* chit;
    float4* lrq;         // [bounce][cap], 2 per entry
    uint4* lhit;
    float4 *lpos, *lrad, *lw, *lpre, *lq;  // [bounce][path]
    float4* conn;        // connections of one bounce: light vertex and path, camera vertex and record
    uint32_t* conn_v;    // their light vertex number
    uint32_t* seen;      // the unoccluded ones
};

// ------------------------------------------------------------ paths ---
// What a path needs of its job, and its pixel's derivative over the samples.
struct AdjPath {
    const AdjJob* J;
    uint32_t pixel, sample;
};
__device__ __forceinline__ AdjPath adj_path(const AdjWave& A, int k)
{
    AdjPath p;
    p.J = A.jobs + (A.path_job ? A.path_job[k] : 0u);
    const int64_t local = A.wave_base + k - p.J->path_base;
    const uint32_t spp = (uint32_t)p.J->spp;
    if (local <= (int64_t)0xFFFFFFFFu) {
        p.pixel = fast_div(p.J->spp_div, (uint32_t)local);
        p.sample = (uint32_t)local - p.pixel * spp;
    } else {
        p.pixel = (uint32_t)(local / spp);
        p.sample = (uint32_t)(local % spp);
    }
    p.sample += (uint32_t)p.J->sample_offset;
    return p;
}
__device__ __forceinline__ V3 adj_delta(const AdjPath& p)
{
    const float* ad = p.J->adj + 3 * (size_t)p.pixel;
    const float s = p.J->inv_spp;
    return v3(ad[0] * s, ad[1] * s, ad[2] * s);
}
__device__ __forceinline__ bool is_zero(V3 a) { return a.x == 0.0f && a.y == 0.0f && a.z == 0.0f; }

// ------------------------------------------------- gradient sums ---
// a term of a gradient unless it is not finite: a degenerate path (an infinite
// sample of the forward estimator) must not poison the sum
__device__ __forceinline__ float finite_or_zero(float t) { return fabsf(t) <= kFltMax ? t : 0.0f; }

// A vertex's terms sum_c a[c] * g.d[c][i] for the parameter slots of its
// material: `key` the first of six consecutive sums (-1: none).  PBR: slots
// 0-4 (the sixth adds zero), OpenMATERIAL: slots 5-10.
struct GradTerms {
    int key;
    float v[6];
};
__device__ __forceinline__ void no_terms(GradTerms& t)
{
    t.key = -1;
#pragma unroll
    for (int i = 0; i < 6; ++i) t.v[i] = 0.0f;
}
__device__ __forceinline__ float channel(V3 a, int c) { return c == 0 ? a.x : c == 1 ? a.y : a.z; }

// key of the material's sums; false for the missing material, which has no
// parameters
__device__ __forceinline__ bool terms_key(GradTerms& t, const AdjJob& J, const DevMaterial& M, uint32_t mat)
{
    const uint32_t m = mat - J.mat_base;
    if (m >= (uint32_t)J.nmat || M.type == kMatMissing) return false;
    t.key = J.key_base + (int)m * kSlots + (M.type == kMatOm ? 5 : 0);
    return true;
}
// a channel's terms: its adjoint a times its derivatives
__device__ __forceinline__ void pbr_terms(GradTerms& t, int c, float a, float rough, Dual<3> f)
{
    const float col = finite_or_zero(a * f.d[0]);
    t.v[0] += c == 0 ? col : 0.0f;
    t.v[1] += c == 1 ? col : 0.0f;
    t.v[2] += c == 2 ? col : 0.0f;
    t.v[3] += finite_or_zero(a * f.d[1] * 2.0f * rough);  // alpha = roughness^2
    t.v[4] += finite_or_zero(a * f.d[2]);
}
__device__ __forceinline__ void om_terms(GradTerms& t, int c, float a, Dual<2> f)
{
    const float n = finite_or_zero(a * f.d[0]), k = finite_or_zero(a * f.d[1]);
    t.v[0] += c == 0 ? n : 0.0f;
    t.v[1] += c == 1 ? n : 0.0f;
    t.v[2] += c == 2 ? n : 0.0f;
    t.v[3] += c == 0 ? k : 0.0f;
    t.v[4] += c == 1 ? k : 0.0f;
    t.v[5] += c == 2 ? k : 0.0f;
}

// The terms of a sampled weight (material_sample times the cosine of `out` or,
// for a light vertex, of `in`; directions fixed) against its adjoint a.
__device__ __forceinline__ void sample_terms(GradTerms& t, const AdjJob& J, const DevScene& S, const DevMaterial& M,
                                             const Surf& sp, uint32_t mat, V3 in, bool light, const Rng4& u, V3 a)
{
    SampleInfo info;
    V3 out;
    const V3 w = material_sample(S, M, sp, in, !light, u, out, &info);
    const float ct = fabsf(dot(light ? in : out, sp.nrm));
    if (M.type == kMatPbr) {
        if (info.kind < 0 || !terms_key(t, J, M, mat)) return;
        const float alpha = M.alpha, metal = M.metal, rough = sqrtf(alpha);
        const DualEvaluate e = d_bsdf_evaluate(in, out, info.N, alpha, info.kind, info.H, info.p);
        const float score = info.kind != 0 ? ggx_log_pdf_dalpha(fabsf(dot(info.N, info.H)), alpha) : 0.0f;
#pragma unroll 1
        for (int c = 0; c < 3; ++c) {
            Dual<3> f = d_evaluate_channel(e, M.color[c], metal);
            f.d[1] += channel(w, c) * score;
#pragma unroll
            for (int i = 0; i < 3; ++i) f.d[i] *= ct;
            pbr_terms(t, c, channel(a, c), rough, f);
        }
    } else if (M.type == kMatOm && M.om_valid) {
        if (!terms_key(t, J, M, mat)) return;
        const float cth = dot(out, sp.nrm);
#pragma unroll 1
        for (int c = 0; c < 3; ++c) {
            Dual<2> f = d_om_channel(M.om_n[c], M.om_k[c], cth);
            f.d[0] *= ct;
            f.d[1] *= ct;
            om_terms(t, c, channel(a, c), f);
        }
    }
}

// material_eval, and its terms against its adjoint a
__device__ __forceinline__ V3 eval_terms(GradTerms& t, const AdjJob& J, const DevMaterial& M, const Surf& sp,
                                         uint32_t mat, V3 in, V3 out, V3 a)
{
    const V3 f = material_eval(M, sp, in, out);
    if (M.type == kMatPbr) {
        if (!terms_key(t, J, M, mat)) return f;
        V3 N = sp.nrm;
        if (dot(in, N) > 0.0f && M.transmissive) N = -N;
        const float alpha = M.alpha, metal = M.metal, rough = sqrtf(alpha);
        const DualDirect e = d_bsdf_eval_direct(in, out, N, alpha);
#pragma unroll 1
        for (int c = 0; c < 3; ++c) pbr_terms(t, c, channel(a, c), rough, d_direct_channel(e, M.color[c], metal));
    } else if (M.type == kMatOm && M.om_valid) {
        const float cth = -dot(in, sp.nrm);
        if (fabsf(dot(out, sp.nrm) - cth) > 1e-6f || !terms_key(t, J, M, mat)) return f;
#pragma unroll 1
        for (int c = 0; c < 3; ++c) om_terms(t, c, channel(a, c), d_om_channel(M.om_n[c], M.om_k[c], cth));
    }
    return f;
}

// Adds the lanes' terms to the warp's sums; every lane of the warp calls it.
// The lanes of one material pair up and halve until its first lane holds their
// total (reduction among a warp's peers: E. Westphal, "Voting and shuffling to
// optimize atomic operations", NVIDIA developer blog, 2015): at most five rounds for all materials at once, where a full reduction
// per material in the warp takes up to eight times thirty shuffles (the replay
// of 512x512x32: 9.54 ms so, 9.44 with pairs).
__device__ __forceinline__ void add_terms(float* sums, GradTerms t)
{
    const int lane = threadIdx.x & 31;
    if (!__any_sync(0xFFFFFFFFu, t.key >= 0)) return;
    const uint32_t same = __match_any_sync(0xFFFFFFFFu, t.key);
    uint32_t rank = __popc(same & ((1u << lane) - 1u));
    const bool first = rank == 0u;
    uint32_t later = same & ~((2u << lane) - 1u);
    while (__any_sync(0xFFFFFFFFu, later != 0u)) {
        const int from = (__ffs(later) - 1) & 31;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const float x = __shfl_sync(0xFFFFFFFFu, t.v[i], from);
            if (later) t.v[i] += x;
        }
        later &= __ballot_sync(0xFFFFFFFFu, !(rank & 1u));
        rank >>= 1;
    }
    if (first && t.key >= 0) {
#pragma unroll
        for (int i = 0; i < 6; ++i) sums[t.key + i] += t.v[i];
    }
    __syncwarp();
}

// the warps' sums of a block: cleared before, added to the wave's after
__device__ __forceinline__ float* clear_sums(float* shared, int keys)
{
    for (int i = threadIdx.x; i < keys * (kAdjThreads / 32); i += kAdjThreads) shared[i] = 0.0f;
    __syncthreads();
    return shared + (threadIdx.x >> 5) * keys;
}
__device__ __forceinline__ void flush_sums(const float* shared, const AdjWave& A)
{
    __syncthreads();
    for (int i = threadIdx.x; i < A.keys; i += kAdjThreads) {
        float x = 0.0f;
#pragma unroll
        for (int w = 0; w < kAdjThreads / 32; ++w) x += shared[w * A.keys + i];
        if (x != 0.0f) atomicAdd(A.acc + i, (double)x);
    }
}

// ------------------------------------------------------------ setup ---
__global__ void k_adj_put_jobs(AdjJobChunk c, AdjJob* table, int first, int n)
{
    const int i = threadIdx.x;
    if (i < n) table[first + i] = c.j[i];
}

// job of every path of the wave (largest job whose first path <= g)
__global__ void __launch_bounds__(kShadeThreads) k_adj_path_jobs(AdjWave A)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= A.wave_n) return;
    const int64_t g = A.wave_base + k;
    int lo = 0, hi = A.num_jobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (A.jobs[mid].path_base <= g)
            lo = mid;
        else
            hi = mid - 1;
    }
    A.path_job[k] = (uint32_t)lo;
}

// Paths of pixels without a derivative add nothing: they are not queued.
// (k_light_gen)
__global__ void __launch_bounds__(kShadeThreads) k_adj_light_gen(AdjWave A)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    bool live = false;
    V3 so = v3(0, 0, 0), R = v3(0, 0, 1);
    if (k < A.wave_n) {
        const AdjPath p = adj_path(A, k);
        const AdjJob& J = *p.J;
        if (!is_zero(adj_delta(p))) {
            int li = J.light_base;
            if (J.light_count > 1)
                li += pick_light(A.S.light_cdf + J.light_base, J.light_count,
                                 rng4(J.seed, p.pixel, p.sample, 0u, kStreamLight).u[0] * J.light_max);
            A.lmeta[k] = (uint32_t)li;
            A.lsuffix[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            live = A.light_bounces >= 1;
            if (live) {
                R = light_direction(J.seed, p.pixel, p.sample);
                const float4 lp = __ldg(A.S.light_pos + li);
                so = shifted_origin(v3(lp.x, lp.y, lp.z), R, 1.0f);
            }
        }
    }
    const uint32_t slot = warp_append(A.ctr + kAdjCtrLight, live);
    if (live) {
        A.lrq[2 * (size_t)slot] = make_float4(so.x, so.y, so.z, 0.0f);
        A.lrq[2 * (size_t)slot + 1] = make_float4(R.x, R.y, R.z, __int_as_float(k));
    }
}

// (k_camera_gen)
__global__ void __launch_bounds__(kShadeThreads) k_adj_camera_gen(AdjWave A)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    bool live = false;
    V3 so = v3(0, 0, 0), R = v3(0, 0, 1);
    if (k < A.wave_n) {
        const AdjPath p = adj_path(A, k);
        live = !is_zero(adj_delta(p));
        if (live) {
            const AdjJob& J = *p.J;
            const Rng4 r = rng4(J.seed, p.pixel, p.sample, 0u, kStreamCamera);
            const uint32_t row = fast_div(J.width_div, p.pixel);
            V3 O;
            camera_ray(J.cam, (int)(p.pixel - row * (uint32_t)J.cam.width), (int)row, r.u[0], r.u[1], O, R);
            so = shifted_origin(O, R, 1.0f);
        }
    }
    const uint32_t slot = warp_append(A.ctr + kAdjCtrCam, live);
    if (live) {
        A.crq[2 * (size_t)slot] = make_float4(so.x, so.y, so.z, 0.0f);
        A.crq[2 * (size_t)slot + 1] = make_float4(R.x, R.y, R.z, __int_as_float(k));
    }
}

// ----------------------------------------------------------- tracing ---
__device__ __forceinline__ uint32_t adj_root(const AdjWave& A, int k)
{
    return A.jobs[A.path_job ? A.path_job[k] : 0u].tlas_root;
}

__global__ void __launch_bounds__(kTraceThreads, kTraceMinBlocks)
    k_adj_extend(const __grid_constant__ AdjWave A, float4* rq, uint4* hits, const uint32_t* count, uint32_t* work)
{
    __shared__ uint2 sstack[kStackShared * kTraceThreads];
    TraceStack st;
    st.sh = sstack + threadIdx.x;
    st.stride = kTraceThreads;
    st.overflow = 0;
    TraceCounters tc{0u, 0u};
    const AdjJob* jobs = A.jobs;
    const uint32_t* path_job = A.path_job;
    auto root = [=](int k) { return jobs[path_job ? path_job[k] : 0u].tlas_root; };
    const uint32_t n = *count;
    if (n <= kCoopRays)
        extend_rays_coop(A.S, A.items, rq, hits, n, work, sstack, root);
    else
        extend_rays(A.S, A.items, rq, hits, n, work, st, tc, root);
}

// k_adj_shadow's loop for short queues, eight lanes per connection
template <bool kMasked>
__device__ __noinline__ void adj_shadow_coop(const AdjWave& A, uint32_t n, uint32_t* seen, uint32_t* work, uint2* stacks)
{
    CoopGroup g = coop_group(stacks);
    TraceCounters tc{0u, 0u};
    TraceStack unused;
    for (RayShares s = ray_shares(32u / kCoopLanes, n); s.next < n; next_step(s, 32u / kCoopLanes, n, work)) {
        const uint32_t base = s.next;
        const uint32_t i = base + (uint32_t)g.index;
        bool ok = false;
        if (i < n) {
            const float4 q0 = A.conn[2 * (size_t)i], q1 = A.conn[2 * (size_t)i + 1];
            ok = is_connected<kMasked>(A.S, A.items, v3(q0.x, q0.y, q0.z), v3(q1.x, q1.y, q1.z), unused, tc,
                                       adj_root(A, __float_as_int(q0.w)), &g) &&
                 g.sub == 0;
        }
        const uint32_t slot = warp_append(seen, ok);
        if (ok) A.seen[slot] = i;
    }
}

// the connections of one camera bounce: the unoccluded ones are listed
template <bool kMasked>
__global__ void __launch_bounds__(kTraceThreads, kTraceMinBlocks)
    k_adj_shadow(const __grid_constant__ AdjWave A, const uint32_t* count, uint32_t* seen, uint32_t* work)
{
    __shared__ uint2 sstack[kStackShared * kTraceThreads];
    TraceStack st;
    st.sh = sstack + threadIdx.x;
    st.stride = kTraceThreads;
    st.overflow = 0;
    TraceCounters tc{0u, 0u};
    const uint32_t n = *count;
    const int lane = threadIdx.x & 31;
    if (n <= kCoopRays) {
        adj_shadow_coop<kMasked>(A, n, seen, work, sstack);
        return;
    }
    for (RayShares s = ray_shares(32u, n); s.next < n; next_step(s, 32u, n, work)) {
        const uint32_t base = s.next;
        const uint32_t i = base + lane;
        bool ok = false;
        if (i < n) {
            const float4 q0 = A.conn[2 * (size_t)i], q1 = A.conn[2 * (size_t)i + 1];
            ok = is_connected<kMasked>(A.S, A.items, v3(q0.x, q0.y, q0.z), v3(q1.x, q1.y, q1.z), st, tc,
                                       adj_root(A, __float_as_int(q0.w)));
        }
        const uint32_t slot = warp_append(seen, ok);
        if (ok) A.seen[slot] = i;
    }
}

// ----------------------------------------------------------- forward ---
// Light vertex b of every queued path (light_vertex, k_light_shade): the
// connection end point, its weight and the product before it, the next ray.
__global__ void __launch_bounds__(kShadeThreads, 4) k_adj_light(AdjWave A, int b)
{
    const DevScene& S = A.S;
    const size_t off = (size_t)(b - 1) * A.cap;
    const float4* rq = A.lrq + 2 * off;
    const uint4* hits = A.lhit + off;
    const uint32_t n = A.ctr[kAdjCtrLight + b - 1];
    for (uint32_t i0 = blockIdx.x * blockDim.x; i0 < n; i0 += gridDim.x * blockDim.x) {
        const uint32_t i = i0 + threadIdx.x;
        bool push = false;
        V3 so = v3(0, 0, 0), O = v3(0, 0, 1);
        float tnear = 0.0f;
        int k = 0;
        const uint4 h = i < n ? hits[i] : make_uint4(kInvalid, 0u, 0u, 0u);
        if (h.x != kInvalid) {
            const float4 ra = rq[2 * (size_t)i], rb = rq[2 * (size_t)i + 1];
            k = __float_as_int(rb.w);
            tnear = ra.w;
            const AdjPath p = adj_path(A, k);
            const AdjJob& J = *p.J;
            const DevMaterial& M = J.mats[__ldg(&S.insts[h.x].material)];
            const Surf sp = surface_point(S, h.x, h.y, __uint_as_float(h.z), __uint_as_float(h.w), true, &M);
            const V3 R = v3(rb.x, rb.y, rb.z);
            const Rng4 u = rng4(J.seed, p.pixel, p.sample, kDimLightBounce + (uint32_t)b, kStreamLight);
            const V3 brdf = material_sample(S, M, sp, R, false, u, O);
            const float ct = fabsf(dot(R, sp.nrm));
            const uint32_t li = A.lmeta[k] & kLightMask;
            const float4 I = __ldg(S.light_int + li);
            const V3 rad0 = v3(I.x * A.light_scale, I.y * A.light_scale, I.z * A.light_scale);
            V3 ltp = v3(1.0f, 1.0f, 1.0f);
            float att;
            if (b == 1) {
                const float4 lp = __ldg(S.light_pos + li);
                const V3 dd = sp.pos - v3(lp.x, lp.y, lp.z);
                att = light_attenuation(A.atten_mode, A.min_dist, sqrtf(dot(dd, dd)), lp.w);
            } else {
                const float4 t = A.ltp[k];
                ltp = v3(t.x, t.y, t.z);
                att = t.w;
            }
            const V3 tp = v3(ltp.x * brdf.x * ct, ltp.y * brdf.y * ct, ltp.z * brdf.z * ct);
            const V3 orad = v3(tp.x * rad0.x * att, tp.y * rad0.y * att, tp.z * rad0.z * att);
            if (!(intensity(orad) < A.cut)) {
                const size_t v = off + k;
                A.lpos[v] = make_float4(sp.pos.x, sp.pos.y, sp.pos.z, 0.0f);
                A.lrad[v] = make_float4(orad.x, orad.y, orad.z, 0.0f);
                A.lw[v] = make_float4(brdf.x * ct, brdf.y * ct, brdf.z * ct, 0.0f);
                A.lpre[v] = make_float4(ltp.x * rad0.x * att, ltp.y * rad0.y * att, ltp.z * rad0.z * att, 0.0f);
                A.lq[v] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                A.lmeta[k] = li | ((uint32_t)b << kLenShift);
                A.ltp[k] = make_float4(tp.x, tp.y, tp.z, att);
                push = b < A.light_bounces && !is_zero(tp);
                if (push) so = shifted_origin(sp.pos, O, 1.0f);
            }
        }
        const uint32_t slot = warp_append(A.ctr + kAdjCtrLight + b, push);
        if (push) {
            float4* out = A.lrq + 2 * (off + A.cap + slot);
            out[0] = make_float4(so.x, so.y, so.z, tnear);
            out[1] = make_float4(O.x, O.y, O.z, __int_as_float(k));
        }
    }
}

// the radiance and direction cosine of the connection from light vertex v of
// path k (position lPos, direction LC to the camera vertex)
__device__ __forceinline__ V3 connection_radiance(const AdjWave& A, uint32_t li, int v, int k, V3 pos, V3 lPos)
{
    if (v > 0) {
        const float4 r = A.lrad[(size_t)(v - 1) * A.cap + k];
        return v3(r.x, r.y, r.z);
    }
    const float4 I = __ldg(A.S.light_int + li);
    const V3 dd = pos - lPos;
    const float f = A.light_scale * light_attenuation(A.atten_mode, A.min_dist, sqrtf(dot(dd, dd)),
                                                      __ldg(A.S.light_pos + li).w);
    return v3(I.x * f, I.y * f, I.z * f);
}

// Camera vertex b of every queued path (camera_vertex, k_camera_shade): its
// record, its candidate connections and the next ray.
__global__ void __launch_bounds__(kShadeThreads, 4) k_adj_camera(AdjWave A, int b)
{
    __shared__ BinScratch bins;
    const DevScene& S = A.S;
    const size_t off = (size_t)(b - 1) * A.cap;
    const float4* rq = A.crq + 2 * off;
    const uint32_t n = A.ctr[kAdjCtrCam + b - 1];
    for (uint32_t i0 = blockIdx.x * blockDim.x; i0 < n; i0 += gridDim.x * blockDim.x) {
        const uint32_t i = i0 + threadIdx.x;
        bool push = false;
        V3 so = v3(0, 0, 0), O = v3(0, 0, 1), tpn = v3(0, 0, 0);
        float tnear = 0.0f;
        int k = 0;
        if (i < n) {
            const float4 ra = rq[2 * (size_t)i], rb = rq[2 * (size_t)i + 1];
            const uint4 h = A.chit[off + i];
            k = __float_as_int(rb.w);
            tnear = ra.w;
            const V3 in = v3(rb.x, rb.y, rb.z);
            V3 G = v3(0.0f, 0.0f, 0.0f);
            // the throughput: 1, or left by the previous bounce
            const float4 tp4 = b == 1 ? make_float4(1.0f, 1.0f, 1.0f, 0.0f) : A.ctp[off + i];
            const V3 tp = v3(tp4.x, tp4.y, tp4.z);
            if (h.x == kInvalid) {
                if (S.env.present && b <= A.max_len) G = env_radiance(S.env, in);
            } else {
                const AdjPath p = adj_path(A, k);
                const AdjJob& J = *p.J;
                const DevMaterial& M = J.mats[__ldg(&S.insts[h.x].material)];
                const Surf sp = surface_point(S, h.x, h.y, __uint_as_float(h.z), __uint_as_float(h.w), true, &M);
                const Rng4 u = rng4(J.seed, p.pixel, p.sample, (uint32_t)b, kStreamCamera);
                const V3 brdf = material_sample(S, M, sp, in, true, u, O);
                const float ct = fabsf(dot(O, sp.nrm));
                if (J.light_count > 0) {
                    const uint32_t meta = A.lmeta[k];
                    const int lp_len = (int)(meta >> kLenShift) + 1;
                    const uint32_t li = meta & kLightMask;
                    for (int v = 0; v < lp_len && v + b <= A.max_len; ++v) {
                        const float4 lp = v == 0 ? __ldg(S.light_pos + li) : A.lpos[(size_t)(v - 1) * A.cap + k];
                        const V3 lPos = v3(lp.x, lp.y, lp.z);
                        const V3 LC = normalize(sp.pos - lPos);
                        const V3 lRad = connection_radiance(A, li, v, k, sp.pos, lPos);
                        const float c = fabsf(dot(LC, sp.nrm));
                        V3 lc = v3(lRad.x * c * tp.x, lRad.y * c * tp.y, lRad.z * c * tp.z);
                        if (intensity(lc) < A.cut) continue;
                        const V3 f = material_eval(M, sp, LC, -in) * c;
                        lc = v3(f.x * tp.x * lRad.x, f.y * tp.y * lRad.y, f.z * tp.z * lRad.z);
                        if (intensity(lc) < A.cut) continue;
                        const uint32_t q = coalesced_append(A.ctr + kAdjCtrConn + b - 1);
                        A.conn[2 * (size_t)q] = make_float4(lPos.x, lPos.y, lPos.z, __int_as_float(k));
                        A.conn[2 * (size_t)q + 1] = make_float4(sp.pos.x, sp.pos.y, sp.pos.z, __uint_as_float(i));
                        A.conn_v[q] = (uint32_t)v;
                    }
                }
                tpn = v3(tp.x * brdf.x * ct, tp.y * brdf.y * ct, tp.z * brdf.z * ct);
                A.cw[off + i] = make_float4(brdf.x * ct, brdf.y * ct, brdf.z * ct, 0.0f);
                push = b < A.cam_bounces && !is_zero(tpn);
                if (push) so = shifted_origin(sp.pos, O, 1.0f);
            }
            A.ctp[off + i] = make_float4(tp.x, tp.y, tp.z, push ? 1.0f : 0.0f);
            A.cG[off + i] = make_float4(G.x, G.y, G.z, 0.0f);
        }
        const uint32_t slot = block_append_binned(A.ctr + kAdjCtrCam + b, push, direction_bin(O), bins);
        if (push) {
            const size_t e = off + A.cap + slot;
            A.crq[2 * e] = make_float4(so.x, so.y, so.z, tnear);
            A.crq[2 * e + 1] = make_float4(O.x, O.y, O.z, __int_as_float(k));
            A.ctp[e] = make_float4(tpn.x, tpn.y, tpn.z, 0.0f);
        }
    }
}

// ---------------------------------------------------------- backward ---
// Every unoccluded connection of camera bounce b: its term of the vertex's G
// and of the light vertex's q, and its derivatives.
__global__ void __launch_bounds__(kAdjThreads) k_adj_connect(AdjWave A, int b)
{
    extern __shared__ float shared_sums[];
    const uint32_t n = A.ctr[kAdjCtrSeen + b - 1];
    if (blockIdx.x * kAdjThreads >= n) return;
    float* sums = clear_sums(shared_sums, A.keys);
    const DevScene& S = A.S;
    const size_t off = (size_t)(b - 1) * A.cap;
    for (uint32_t i0 = blockIdx.x * kAdjThreads; i0 < n; i0 += gridDim.x * kAdjThreads) {
        const uint32_t s = i0 + threadIdx.x;
        GradTerms t;
        no_terms(t);
        if (s < n) {
            const uint32_t q = A.seen[s];
            const float4 q0 = A.conn[2 * (size_t)q], q1 = A.conn[2 * (size_t)q + 1];
            const int v = (int)A.conn_v[q], k = __float_as_int(q0.w);
            const size_t e = off + __float_as_uint(q1.w);
            const uint4 h = A.chit[e];
            const float4 rb = A.crq[2 * e + 1], tp4 = A.ctp[e];
            const V3 lPos = v3(q0.x, q0.y, q0.z), tp = v3(tp4.x, tp4.y, tp4.z);
            const AdjPath p = adj_path(A, k);
            const AdjJob& J = *p.J;
            const uint32_t mat = __ldg(&S.insts[h.x].material);
            const DevMaterial& M = J.mats[mat];
            const Surf sp = surface_point(S, h.x, h.y, __uint_as_float(h.z), __uint_as_float(h.w), true, &M);
            const V3 LC = normalize(sp.pos - lPos);
            const V3 lRad = connection_radiance(A, A.lmeta[k] & kLightMask, v, k, sp.pos, lPos);
            const float c = fabsf(dot(LC, sp.nrm));
            const V3 a = mul(adj_delta(p), tp);
            const V3 f = eval_terms(t, J, M, sp, mat, LC, -v3(rb.x, rb.y, rb.z),
                                    mul(a, v3(lRad.x * c, lRad.y * c, lRad.z * c))) *
                         c;
            const V3 G = mul(f, lRad);
            float* pg = &A.cG[e].x;
            atomicAdd(pg, G.x);
            atomicAdd(pg + 1, G.y);
            atomicAdd(pg + 2, G.z);
            if (v > 0) {
                const V3 dq = mul(a, f);
                float* pq = &A.lq[(size_t)(v - 1) * A.cap + k].x;
                atomicAdd(pq, dq.x);
                atomicAdd(pq + 1, dq.y);
                atomicAdd(pq + 2, dq.z);
            }
        }
        add_terms(sums, t);
    }
    flush_sums(shared_sums, A);
}

// Camera vertices of bounce b, last bounce first: the derivative of the sampled
// weight against the suffix radiance, then the suffix through the vertex.
__global__ void __launch_bounds__(kAdjThreads) k_adj_camera_back(AdjWave A, int b)
{
    extern __shared__ float shared_sums[];
    const uint32_t n = A.ctr[kAdjCtrCam + b - 1];
    if (blockIdx.x * kAdjThreads >= n) return;
    float* sums = clear_sums(shared_sums, A.keys);
    const DevScene& S = A.S;
    const size_t off = (size_t)(b - 1) * A.cap;
    for (uint32_t i0 = blockIdx.x * kAdjThreads; i0 < n; i0 += gridDim.x * kAdjThreads) {
        const uint32_t i = i0 + threadIdx.x;
        GradTerms t;
        no_terms(t);
        if (i < n) {
            const float4 tp4 = A.ctp[off + i], G4 = A.cG[off + i];
            const float4 rb = A.crq[2 * (off + i) + 1];
            const int k = __float_as_int(rb.w);
            V3 R = v3(G4.x, G4.y, G4.z);
            if (tp4.w != 0.0f) {  // the path went on
                const float4 s4 = A.suffix[k], w4 = A.cw[off + i];
                const V3 Rs = v3(s4.x, s4.y, s4.z);
                const AdjPath p = adj_path(A, k);
                const V3 a = mul(mul(adj_delta(p), v3(tp4.x, tp4.y, tp4.z)), Rs);
                if (!is_zero(a)) {
                    const AdjJob& J = *p.J;
                    const uint4 h = A.chit[off + i];
                    const uint32_t mat = __ldg(&S.insts[h.x].material);
                    const DevMaterial& M = J.mats[mat];
                    const Surf sp = surface_point(S, h.x, h.y, __uint_as_float(h.z), __uint_as_float(h.w), true, &M);
                    const Rng4 u = rng4(J.seed, p.pixel, p.sample, (uint32_t)b, kStreamCamera);
                    sample_terms(t, J, S, M, sp, mat, v3(rb.x, rb.y, rb.z), false, u, a);
                }
                R = R + mul(v3(w4.x, w4.y, w4.z), Rs);
            }
            A.suffix[k] = make_float4(R.x, R.y, R.z, 0.0f);
        }
        add_terms(sums, t);
    }
    flush_sums(shared_sums, A);
}

// Light vertices of bounce b, last bounce first.
__global__ void __launch_bounds__(kAdjThreads) k_adj_light_back(AdjWave A, int b)
{
    extern __shared__ float shared_sums[];
    const uint32_t n = A.ctr[kAdjCtrLight + b - 1];
    if (blockIdx.x * kAdjThreads >= n) return;
    float* sums = clear_sums(shared_sums, A.keys);
    const DevScene& S = A.S;
    const size_t off = (size_t)(b - 1) * A.cap;
    for (uint32_t i0 = blockIdx.x * kAdjThreads; i0 < n; i0 += gridDim.x * kAdjThreads) {
        const uint32_t i = i0 + threadIdx.x;
        GradTerms t;
        no_terms(t);
        const uint4 h = i < n ? A.lhit[off + i] : make_uint4(kInvalid, 0u, 0u, 0u);
        if (h.x != kInvalid) {
            const float4 rb = A.lrq[2 * (off + i) + 1];
            const int k = __float_as_int(rb.w);
            if ((int)(A.lmeta[k] >> kLenShift) >= b) {  // the vertex was kept (its radiance passed the cutoff)
                const size_t v = off + k;
                const float4 q4 = A.lq[v], s4 = A.lsuffix[k], pre = A.lpre[v], w4 = A.lw[v];
                const V3 Ss = v3(q4.x + s4.x, q4.y + s4.y, q4.z + s4.z);
                A.lsuffix[k] = make_float4(w4.x * Ss.x, w4.y * Ss.y, w4.z * Ss.z, 0.0f);
                const V3 a = mul(v3(pre.x, pre.y, pre.z), Ss);
                if (!is_zero(a)) {
                    const AdjPath p = adj_path(A, k);
                    const AdjJob& J = *p.J;
                    const uint32_t mat = __ldg(&S.insts[h.x].material);
                    const DevMaterial& M = J.mats[mat];
                    const Surf sp = surface_point(S, h.x, h.y, __uint_as_float(h.z), __uint_as_float(h.w), true, &M);
                    const Rng4 u = rng4(J.seed, p.pixel, p.sample, kDimLightBounce + (uint32_t)b, kStreamLight);
                    sample_terms(t, J, S, M, sp, mat, v3(rb.x, rb.y, rb.z), true, u, a);
                }
            }
        }
        add_terms(sums, t);
    }
    flush_sums(shared_sums, A);
}

// the wave loop's sums to the callers' buffers (which may be shared by jobs)
__global__ void k_adj_out(AdjWave A)
{
    for (int j = 0; j < A.num_jobs; ++j) {
        const AdjJob& J = A.jobs[j];
        for (int i = threadIdx.x; i < J.nmat * kSlots; i += blockDim.x) {
            const float x = (float)A.acc[J.key_base + i];
            if (x != 0.0f) atomicAdd(J.grad + i, x);
        }
    }
}

// -------------------------------------------------------------- host ---
// Byte offsets of a wave's arrays in one block (each on a 256-byte boundary).
struct AdjLayout {
    size_t ctr, acc, jobs, path_job, suffix, lmeta, ltp, lsuffix, crq, ctp, cw, cG, chit, lrq, lhit, lpos, lrad, lw,
        lpre, lq, conn, conn_v, seen, bytes;
};
AdjLayout adj_layout(int64_t cap, int njobs, int B, int L, bool lights)
{
    const size_t W = (size_t)cap, cb = (size_t)std::max(B, 1), lb = lights ? (size_t)std::max(L, 1) : 0;
    const size_t lw = lights ? W : 0, slots = lights ? (size_t)L + 1 : 0;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off += (bytes + 255) & ~(size_t)255;
        return o;
    };
    AdjLayout l;
    l.ctr = take(kAdjCounters * 4);
    l.acc = take(kAdjMaxKeys * 8);
    l.jobs = take(sizeof(AdjJob) * (size_t)njobs);
    l.path_job = take(njobs > 1 ? W * 4 : 0);
    l.suffix = take(W * 16);
    l.lmeta = take(lw * 4);
    l.ltp = take(lw * 16);
    l.lsuffix = take(lw * 16);
    l.crq = take(cb * W * 32);
    l.ctp = take(cb * W * 16);
    l.cw = take(cb * W * 16);
    l.cG = take(cb * W * 16);
    l.chit = take(cb * W * 16);
    l.lrq = take(lb * W * 32);
    l.lhit = take(lb * W * 16);
    l.lpos = take(lb * W * 16);
    l.lrad = take(lb * W * 16);
    l.lw = take(lb * W * 16);
    l.lpre = take(lb * W * 16);
    l.lq = take(lb * W * 16);
    l.conn = take(slots * W * 32);
    l.conn_v = take(slots * W * 4);
    l.seen = take(slots * W * 4);
    l.bytes = off;
    return l;
}
void carve_wave(AdjWave& A, char* b, const AdjLayout& l, int njobs)
{
    A.ctr = (uint32_t*)(b + l.ctr);
    A.acc = (double*)(b + l.acc);
    A.jobs = (const AdjJob*)(b + l.jobs);
    A.path_job = njobs > 1 ? (uint32_t*)(b + l.path_job) : nullptr;
    A.suffix = (float4*)(b + l.suffix);
    A.lmeta = (uint32_t*)(b + l.lmeta);
    A.ltp = (float4*)(b + l.ltp);
    A.lsuffix = (float4*)(b + l.lsuffix);
    A.crq = (float4*)(b + l.crq);
    A.ctp = (float4*)(b + l.ctp);
    A.cw = (float4*)(b + l.cw);
    A.cG = (float4*)(b + l.cG);
    A.chit = (uint4*)(b + l.chit);
    A.lrq = (float4*)(b + l.lrq);
    A.lhit = (uint4*)(b + l.lhit);
    A.lpos = (float4*)(b + l.lpos);
    A.lrad = (float4*)(b + l.lrad);
    A.lw = (float4*)(b + l.lw);
    A.lpre = (float4*)(b + l.lpre);
    A.lq = (float4*)(b + l.lq);
    A.conn = (float4*)(b + l.conn);
    A.conn_v = (uint32_t*)(b + l.conn_v);
    A.seen = (uint32_t*)(b + l.seen);
}

// Records of one wave: up to 8 GiB, and at most half of the free memory.  Every
// further wave pays the latency of the last, nearly empty bounces again: a
// 512x512x32 replay with 6 bounces (14 GB of records) takes two waves, 0.17 ms
// more than one wave of 16 GiB would (gradient step 13.10 against 12.93 ms).
constexpr size_t kAdjBudget = (size_t)8 << 30;
constexpr int64_t kAdjMinCap = 1 << 14;  // tried at least, whatever memory is free

// Where a wave's records live while its launches are in flight: a block of the
// context's work memory, for the call or, when the caller captures the stream into a
// graph, claimed for that graph, where one call of the capture and one replay of
// any instance after another use it (the graph waits for and records an external
// event).
struct AdjWorkspace {
    cudaStream_t st;
    WorkBlock direct;
    WorkMemory::Block* captured = nullptr;
    void* base = nullptr;
    int64_t cap = 0;
    AdjWorkspace(SceneHost& s, cudaStream_t st_, int64_t total, int njobs, int B, int L, bool lights) : st(st_)
    {
        const bool capturing = is_captured(st);
        auto need = [&](int64_t c) { return adj_layout(c, njobs, B, L, lights).bytes; };
        const size_t per = std::max<size_t>(1, (need(1 << 20) - need(0)) >> 20);
        const int64_t most = std::min<int64_t>(total, (int64_t)1 << 30);
        cap = std::max<int64_t>(1, std::min<int64_t>(most, (int64_t)(kAdjBudget / per)));
        size_t idle = 0, largest = 0;
        if (!capturing) idle = work_memory(s).idle(&largest);
        if (largest < need(cap)) {
            const OutsideCapture outside;
            size_t free_b = 0, total_b = 0;
            OMV_CUDA(cudaMemGetInfo(&free_b, &total_b));
            const int64_t fit = (int64_t)(std::min(kAdjBudget, (free_b + idle) / 2) / per);
            cap = std::min(cap, std::max<int64_t>(std::min(most, kAdjMinCap), fit));
        }
        for (;;) {
            try {
                if (capturing) {
                    captured = work_memory(s).claim(need(cap), st, &s);
                    base = captured->p;
                } else {
                    base = direct.take(work_memory(s), need(cap), st);
                }
                break;
            } catch (const DeviceOutOfMemory&) {  // someone else took it meanwhile
                if (cap <= std::min(most, kAdjMinCap)) throw;
                cap = std::max(cap / 2, std::min(most, kAdjMinCap));
            }
        }
        if (captured) {
            if (captured->shared) OMV_CUDA(cudaStreamWaitEvent(st, captured->done, 0));
            OMV_CUDA(cudaStreamWaitEvent(st, captured->replay, cudaEventWaitExternal));
        }
    }
    ~AdjWorkspace()
    {
        if (!captured) return;
        cudaEventRecord(captured->done, st);
        cudaEventRecordWithFlags(captured->replay, st, cudaEventRecordExternal);
    }
    AdjWorkspace(const AdjWorkspace&) = delete;
    AdjWorkspace& operator=(const AdjWorkspace&) = delete;
};

// The side stream of an adjoint (null: its work runs in line).  It is joined
// before the records are given back, also when a launch fails.
struct AdjSide {
    const SceneHost::Side* side;
    cudaStream_t st;
    bool forked = false;
    AdjSide(const SceneHost::Side* s, cudaStream_t main) : side(s), st(main) {}
    ~AdjSide()
    {
        if (!forked) return;
        cudaEventRecord(side->join, side->stream);
        cudaStreamWaitEvent(st, side->join, 0);
    }
    AdjSide(const AdjSide&) = delete;
    AdjSide& operator=(const AdjSide&) = delete;
    cudaStream_t stream() const { return side ? side->stream : st; }
    void fork()
    {
        if (!side) return;
        fork_side(*side, st);
        forked = true;
    }
    void join()
    {
        if (forked) join_side(*side, st);
        forked = false;
    }
};

inline unsigned blocks_for(int64_t n, int t) { return (unsigned)std::max<int64_t>(1, (n + t - 1) / t); }

template <typename K>
int resident_grid(K kernel, int threads, size_t smem, int sms)
{
    int occ = 0;
    OMV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, smem));
    return std::max(1, occ) * sms;
}

// the checked device form of one job
AdjJob make_job(const SceneHost& s, const omv_camera& cam, const omv_params& p, int32_t spp, int32_t sample_offset,
                uint64_t seed, const float* d_adjoint, float* d_grad, int part, const DevMaterial* mats)
{
    if (part < 0 || part >= (int)s.parts.size()) throw ArgError("adjoint scene (part) out of range");
    const ScenePart& P = s.parts[part];
    if (cam.width <= 0 || cam.height <= 0) throw ArgError("camera resolution must be positive");
    if (spp <= 0) throw ArgError("the adjoint needs at least one sample per pixel");
    if (p.camera_bounces < 0 || p.light_bounces < 0) throw ArgError("negative bounce count");
    if (p.camera_bounces >= kAdjMaxVerts || p.light_bounces >= kAdjMaxVerts)
        throw ArgError("the adjoint supports at most 15 camera and 15 light bounces");
    if (P.mat_count > kAdjMaxMaterials) throw ArgError("the adjoint supports at most 16 materials per scene");
    if (!d_adjoint || !d_grad) throw ArgError("adjoint image and gradient buffers are required");
    if (p.estimator != OMV_ESTIMATOR_REFERENCE) throw ArgError("the adjoint replays the reference estimator only");
    for (const DevMaterial& m : s.h_mats)
        if (m.type == kMatPbr && (m.textured || m.emissive_on))
            throw ArgError("the adjoint differentiates untextured materials only");
    AdjJob J{};
    J.cam = cam;
    J.seed = seed;
    J.mats = mats ? mats : s.dev.mats;
    J.adj = d_adjoint;
    J.grad = d_grad;
    J.spp = spp;
    J.sample_offset = sample_offset;
    J.spp_div = make_fastdiv((uint32_t)spp);
    J.width_div = make_fastdiv((uint32_t)cam.width);
    J.inv_spp = 1.0f / (float)spp;
    J.tlas_root = P.tlas_root;
    J.light_base = P.light_base;
    J.light_count = P.light_count;
    J.light_max = P.light_max;
    J.mat_base = (uint32_t)P.mat_base;
    J.nmat = P.mat_count;
    return J;
}

// The replay of jobs [0, n) as one sequence of waves.
void run_adjoint(SceneHost& s, std::vector<AdjJob>& jobs, const omv_params& p, cudaStream_t st)
{
    int64_t total = 0;
    int keys = 0;
    bool lights = false;
    for (AdjJob& J : jobs) {
        J.path_base = total;
        J.key_base = keys;
        total += (int64_t)J.cam.width * J.cam.height * J.spp;
        keys += J.nmat * kSlots;
        lights = lights || J.light_count > 0;
    }
    if (keys == 0 || p.camera_bounces == 0) return;  // no parameter, or no vertex to differentiate
    bool masked = false;
    for (const DevMaterial& m : s.h_mats) masked = masked || m.masked != 0;
    const int nj = (int)jobs.size(), B = p.camera_bounces, L = p.light_bounces;
    std::lock_guard<std::mutex> lock(s.adj_mutex);
    AdjWorkspace ws(s, st, total, nj, B, L, lights);
    AdjWave A{};
    const AdjLayout lay = adj_layout(ws.cap, nj, B, L, lights);
    carve_wave(A, static_cast<char*>(ws.base), lay, nj);
    A.S = s.dev;
    A.items = s.tlas_items;
    A.num_jobs = nj;
    A.cap = (int32_t)ws.cap;
    A.keys = keys;
    A.cam_bounces = B;
    A.light_bounces = L;
    A.max_len = p.max_path_length;
    A.atten_mode = p.light_distance_attenuation;
    A.light_scale = p.light_scale;
    A.min_dist = p.light_min_distance;
    A.cut = p.ray_cut_value;
    for (int f = 0; f < nj; f += kJobsPerPut) {
        AdjJobChunk c;
        const int m = std::min(kJobsPerPut, nj - f);
        for (int i = 0; i < m; ++i) c.j[i] = jobs[f + i];
        k_adj_put_jobs<<<1, 32, 0, st>>>(c, const_cast<AdjJob*>(A.jobs), f, m);
    }
    OMV_CUDA(cudaMemsetAsync(A.acc, 0, sizeof(double) * keys, st));
    const size_t smem = sizeof(float) * (size_t)keys * (kAdjThreads / 32);
    const int trace_grid = resident_grid(k_adj_extend, kTraceThreads, 0, s.num_sms);
    const int light_grid = resident_grid(k_adj_light, kShadeThreads, 0, s.num_sms);
    const int camera_grid = resident_grid(k_adj_camera, kShadeThreads, 0, s.num_sms);
    const int connect_grid = resident_grid(k_adj_connect, kAdjThreads, smem, s.num_sms);
    const int back_grid = resident_grid(k_adj_camera_back, kAdjThreads, smem, s.num_sms);
    const int lback_grid = resident_grid(k_adj_light_back, kAdjThreads, smem, s.num_sms);
    // beside the main stream: the light subpaths beside the camera rays' first
    // hits, then each bounce's connections beside the next bounce's hits
    AdjSide beside(lights ? side_of(s.adj_side, st) : nullptr, st);
    const cudaStream_t side = beside.stream();
    for (int64_t wb = 0; wb < total; wb += ws.cap) {
        A.wave_base = wb;
        A.wave_n = (int32_t)std::min<int64_t>(ws.cap, total - wb);
        OMV_CUDA(cudaMemsetAsync(A.ctr, 0, kAdjCounters * 4, st));
        uint32_t* work = A.ctr + kAdjCtrWork;
        const unsigned gen = blocks_for(A.wave_n, kShadeThreads);
        if (A.path_job) k_adj_path_jobs<<<gen, kShadeThreads, 0, st>>>(A);
        if (lights) {
            beside.fork();
            k_adj_light_gen<<<gen, kShadeThreads, 0, side>>>(A);
            for (int b = 1; b <= L; ++b) {
                const size_t off = (size_t)(b - 1) * A.cap;
                k_adj_extend<<<trace_grid, kTraceThreads, 0, side>>>(A, A.lrq + 2 * off, A.lhit + off,
                                                                     A.ctr + kAdjCtrLight + b - 1, work++);
                k_adj_light<<<light_grid, kShadeThreads, 0, side>>>(A, b);
            }
        }
        k_adj_camera_gen<<<gen, kShadeThreads, 0, st>>>(A);
        for (int b = 1; b <= B; ++b) {
            const size_t off = (size_t)(b - 1) * A.cap;
            k_adj_extend<<<trace_grid, kTraceThreads, 0, st>>>(A, A.crq + 2 * off, A.chit + off,
                                                               A.ctr + kAdjCtrCam + b - 1, work++);
            beside.join();
            k_adj_camera<<<camera_grid, kShadeThreads, 0, st>>>(A, b);
            if (lights) {
                uint32_t* seen = A.ctr + kAdjCtrSeen + b - 1;
                const uint32_t* count = A.ctr + kAdjCtrConn + b - 1;
                beside.fork();
                if (masked)
                    k_adj_shadow<true><<<trace_grid, kTraceThreads, 0, side>>>(A, count, seen, work++);
                else
                    k_adj_shadow<false><<<trace_grid, kTraceThreads, 0, side>>>(A, count, seen, work++);
                k_adj_connect<<<connect_grid, kAdjThreads, smem, side>>>(A, b);
            }
        }
        beside.join();
        for (int b = B; b >= 1; --b) k_adj_camera_back<<<back_grid, kAdjThreads, smem, st>>>(A, b);
        if (lights)
            for (int b = L; b >= 1; --b) k_adj_light_back<<<lback_grid, kAdjThreads, smem, st>>>(A, b);
        OMV_CUDA(cudaGetLastError());
    }
    k_adj_out<<<1, 256, 0, st>>>(A);
    OMV_CUDA(cudaGetLastError());
}

}  // namespace

void adjoint_frame(SceneHost& s, const omv_camera& cam, const omv_params& p, const float* d_adjoint, float* d_grad,
                   cudaStream_t st)
{
    std::vector<AdjJob> jobs{
        make_job(s, cam, p, p.samples_per_pixel, p.sample_offset, p.seed, d_adjoint, d_grad, 0, nullptr)};
    run_adjoint(s, jobs, p, st);
}

void adjoint_batch(SceneHost& s, int n, const omv_adjoint_job* jobs, const omv_params& p, cudaStream_t st)
{
    std::vector<AdjJob> all;
    all.reserve(n);
    for (int i = 0; i < n; ++i) {  // checked before anything is enqueued
        const omv_job& j = jobs[i].job;
        if (j.material_set < -1 || j.material_set >= s.num_mat_sets)
            throw ArgError("adjoint job material set out of range");
        if (j.part < 0 || j.part >= (int)s.parts.size()) throw ArgError("adjoint job scene (part) out of range");
        if (j.samples_per_pixel <= 0 || j.camera.width <= 0 || j.camera.height <= 0)
            throw ArgError("adjoint job without samples or pixels");
        if (!jobs[i].d_adjoint_rgb || !jobs[i].d_grad) throw ArgError("adjoint job without adjoint image or gradient");
        const DevMaterial* mats = j.material_set < 0 ? nullptr : s.mat_sets + (size_t)j.material_set * s.num_materials;
        all.push_back(make_job(s, j.camera, p, j.samples_per_pixel, j.sample_offset, j.seed, jobs[i].d_adjoint_rgb,
                               jobs[i].d_grad, j.part, mats));
    }
    // as many jobs per sequence of waves as the gradient sums have room for
    for (size_t i = 0; i < all.size();) {
        std::vector<AdjJob> group;
        int keys = 0;
        while (i < all.size() && (group.empty() || keys + all[i].nmat * kSlots <= kAdjMaxKeys)) {
            keys += all[i].nmat * kSlots;
            group.push_back(all[i++]);
        }
        run_adjoint(s, group, p, st);
    }
}

}  // namespace omv
