// Tile lists of the first camera bounce: which subtrees the camera rays of a
// small block of pixels can hit.
//
// A warp follows the beam of a tile (all rays through its pixels) down the two
// levels of the tree, eight lanes per node, and keeps the nodes where the beam
// splits up or meets triangles; the tile's rays start at those nodes instead of
// the scene's root.  Tiles that see no object have an empty list, and their
// rays miss without a node visit.
//
// The beam test is conservative for every ray of the tile.  A camera ray is
// R = M c / |c| with c linear in the pixel position, so the unnormalised
// directions M c over the tile lie between their extremes at its corners, in
// world space and (also linear) in every instance's object space; origins lie
// within the ray shift of the camera's position.  Origins, directions and boxes
// are widened by at least ten times the rounding of the rays' own arithmetic
// (camera_ray, shifted_origin, to_object) and of the box test.  At
// distance u along the unnormalised directions the beam covers
// [omin + u dmin, omax + u dmax] per axis; it meets a box iff some u >= 0
// satisfies all six linear constraints.
#pragma once

#include "omv_device.cuh"
#include "omv_types.h"
#include "trace.cuh"

namespace omv {

constexpr int kTileNodes = 16;  // start nodes of a tile
constexpr int kTileRuns = 8;    // instances they belong to

// Start nodes in runs of one instance (kInvalid: nodes of the top-level tree),
// near runs first, near nodes of a run first.
struct alignas(16) TileList {
    uint32_t num_runs;
    uint32_t pad[3];
    struct Run {
        uint32_t inst;
        uint32_t first, count;
        float t;  // no ray of the tile meets the run's nodes before t
    } run[kTileRuns];
    struct Node {
        uint32_t node;
        float t;
    } node[kTileNodes];
};

static_assert(kTileRuns == 8 && sizeof(TileList) == 16 + 16 * kTileRuns + 8 * kTileNodes,
              "tile_run and push_tile_node read this layout");

// one axis of a beam: position at distance u >= 0 within [omin + u dmin, omax + u dmax]
struct BeamAxis {
    float omin, omax, rmin, rmax;  // reciprocals of dmin and dmax (never 0)
};
struct Beam {
    BeamAxis x, y, z;
};

__device__ __forceinline__ BeamAxis beam_axis(float o, float oerr, float d0, float d1, float d2, float d3, float derr)
{
    const float dmin = fminf(fminf(d0, d1), fminf(d2, d3)) - derr - 1e-20f;
    const float dmax = fmaxf(fmaxf(d0, d1), fmaxf(d2, d3)) + derr + 1e-20f;
    // a bound next to zero moves away from zero, outwards
    const float lo = dmin >= 0.0f && dmin < 1e-18f ? -1e-18f : (dmin < 0.0f && dmin > -1e-18f ? -1e-18f : dmin);
    const float hi = dmax <= 0.0f && dmax > -1e-18f ? 1e-18f : (dmax > 0.0f && dmax < 1e-18f ? 1e-18f : dmax);
    return BeamAxis{o - oerr, o + oerr, 1.0f / lo, 1.0f / hi};
}

// constraints of one axis on u for the box side [lo, hi]
__device__ __forceinline__ void beam_clip(const BeamAxis& a, float lo, float hi, float& ulo, float& uhi)
{
    const float p = (hi - a.omin) * a.rmin;  // omin + u dmin <= hi
    if (a.rmin > 0.0f)
        uhi = fminf(uhi, p);
    else
        ulo = fmaxf(ulo, p);
    const float q = (lo - a.omax) * a.rmax;  // omax + u dmax >= lo
    if (a.rmax > 0.0f)
        ulo = fmaxf(ulo, q);
    else
        uhi = fminf(uhi, q);
}
// whether the beam can meet the box; u: a lower bound of the distance
__device__ __forceinline__ bool beam_meets(const Beam& b, V3 lo, V3 hi, float& u)
{
    float ulo = 0.0f, uhi = kFltMax;
    beam_clip(b.x, lo.x, hi.x, ulo, uhi);
    beam_clip(b.y, lo.y, hi.y, ulo, uhi);
    beam_clip(b.z, lo.z, hi.z, ulo, uhi);
    u = ulo * (1.0f - 1e-5f);
    return !(u > uhi + 1e-5f * fabsf(uhi));
}

// the four corner directions of a tile in world space, the camera's position
// and the error bounds of both
struct TileBeam {
    V3 d[4];
    V3 o;
    float oerr;  // of the position, per axis
    float derr;  // of the directions, per axis
    float cmin;  // smallest |c| over the tile: t >= cmin u
};
__device__ __forceinline__ TileBeam tile_beam(const omv_camera& cam, float x0, float x1, float y0, float y1)
{
    TileBeam t;
    const float(*M)[3] = cam.rotation;
    const float f = cam.focus;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float x = (i & 1) ? x1 : x0, y = (i & 2) ? y1 : y0;
        t.d[i] = v3(M[0][0] * x + M[0][1] * y + M[0][2] * f, M[1][0] * x + M[1][1] * y + M[1][2] * f,
                    M[2][0] * x + M[2][1] * y + M[2][2] * f);
    }
    // the largest sum of magnitudes in a component of M c
    const float ax = fmaxf(fabsf(x0), fabsf(x1)), ay = fmaxf(fabsf(y0), fabsf(y1));
    const float far = fmaxf(fabsf(M[0][0]) * ax + fabsf(M[0][1]) * ay + fabsf(M[0][2] * f),
                            fmaxf(fabsf(M[1][0]) * ax + fabsf(M[1][1]) * ay + fabsf(M[1][2] * f),
                                  fabsf(M[2][0]) * ax + fabsf(M[2][1]) * ay + fabsf(M[2][2] * f)));
    t.derr = 3e-6f * far;
    const float cx = x0 > 0.0f ? x0 : x1 < 0.0f ? x1 : 0.0f, cy = y0 > 0.0f ? y0 : y1 < 0.0f ? y1 : 0.0f;
    t.cmin = sqrtf(cx * cx + cy * cy + cam.focus * cam.focus) * (1.0f - 1e-5f);
    t.o = v3(cam.position[0], cam.position[1], cam.position[2]);
    // the ray shift is 3 epsilon max(|O|, 1) along R; |R| <= far / cmin
    const float r = t.cmin > 0.0f ? far / t.cmin : 0.0f;
    t.oerr = 1e-6f * max_abs(t.o, 1.0f) * fmaxf(r, 1.0f);
    return t;
}

// the beam in world space (inv null) or in an instance's object space
__device__ __forceinline__ Beam make_beam(const TileBeam& t, const float* inv)
{
    float m[12] = {1.0f, 0.0f, 0.0f, 0.0f, 0.0f, 1.0f, 0.0f, 0.0f, 0.0f, 0.0f, 1.0f, 0.0f};
    if (inv) {
#pragma unroll
        for (int k = 0; k < 12; ++k) m[k] = __ldg(inv + k);
    }
    Beam b;
    BeamAxis* ax[3] = {&b.x, &b.y, &b.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float m0 = m[4 * a], m1 = m[4 * a + 1], m2 = m[4 * a + 2], m3 = m[4 * a + 3];
        const float o = m0 * t.o.x + m1 * t.o.y + m2 * t.o.z + m3;
        const float mag = fabsf(m0 * t.o.x) + fabsf(m1 * t.o.y) + fabsf(m2 * t.o.z) + fabsf(m3);
        const float oerr = (fabsf(m0) + fabsf(m1) + fabsf(m2)) * t.oerr + 1e-5f * mag;
        float d[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) d[i] = m0 * t.d[i].x + m1 * t.d[i].y + m2 * t.d[i].z;
        *ax[a] = beam_axis(o, oerr, d[0], d[1], d[2], d[3], (fabsf(m0) + fabsf(m1) + fabsf(m2)) * t.derr);
    }
    return b;
}

// The list of one tile, by one warp.  An entry whose node holds no triangle that
// the beam meets is replaced by the children it meets, while there is room.
// (Replacing only where at most two, or three, children are met, since every ray
// of the tile visits every start node: the 1920x1080x64 sky frame 17.65 (17.41)
// ms, a point-light one 39.7 (39.5); with every replacement 17.10 and 39.15.)
constexpr int kTileThreads = 128;
struct TileEntry {
    uint32_t inst, node;
    float u;
    uint32_t done;
};

__device__ __forceinline__ void tile_list(const DevScene& S, const uint32_t* __restrict__ items, const omv_camera& cam,
                                          uint32_t root, int px0, int px1, int py0, int py1, TileEntry* E, TileList* out)
{
    const int lane = threadIdx.x & 31, g = lane >> 3, sub = lane & 7;
    const TileBeam tb = tile_beam(cam, (float)px0 - cam.half_width, (float)px1 - cam.half_width,
                                  (float)py0 - cam.half_height, (float)py1 - cam.half_height);
    // a camera at its own focus has no beam: its rays start at the root
    const bool beam = tb.cmin > 0.0f && tb.derr <= kFltMax;
    if (lane == 0) E[0] = TileEntry{kInvalid, root, 0.0f, beam ? 0u : 1u};
    int n = 1;
    __syncwarp();
    for (int round = 0; round < 24; ++round) {
        // the first four entries not yet done, one per eight lanes
        const uint32_t open = __ballot_sync(0xFFFFFFFFu, lane < n && !E[lane].done);
        if (!open) break;
        uint32_t m = open;
        for (int k = 0; k < g; ++k) m &= m - 1u;
        const int at = m ? __ffs(m) - 1 : -1;
        bool hit = false, tri = false;
        uint32_t child = 0, inst = kInvalid;
        float u = 0.0f;
        if (at >= 0) {
            const TileEntry e = E[at];
            inst = e.inst;
            const uint4* N = S.nodes + 8 * (size_t)e.node;
            const uint4 w0 = __ldg(N), w1 = __ldg(N + 1);
            const uint16_t* P = reinterpret_cast<const uint16_t*>(N + 2) + sub;
            const uint32_t meta = ((sub < 4 ? w1.z : w1.w) >> (8 * (sub & 3))) & 0xFFu;
            const bool internal = (w0.w >> (24 + sub)) & 1u;
            if (internal || meta != 0u) {
                const Beam b = make_beam(tb, inst == kInvalid ? nullptr : S.insts[inst].inv);
                const float s[3] = {__uint_as_float((w0.w & 0xFFu) << 23), __uint_as_float(((w0.w >> 8) & 0xFFu) << 23),
                                    __uint_as_float(((w0.w >> 16) & 0xFFu) << 23)};
                const float p[3] = {__uint_as_float(w0.x), __uint_as_float(w0.y), __uint_as_float(w0.z)};
                float lo[3], hi[3];
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    const float err = 1e-6f * (fabsf(p[a]) + 32768.0f * s[a]) + 1e-30f;
                    lo[a] = p[a] + (float)(__ldg(P + 8 * a) & kQuantMax) * s[a] - err;
                    hi[a] = p[a] + (float)(__ldg(P + 24 + 8 * a) & kQuantMax) * s[a] + err;
                }
                hit = beam_meets(b, v3(lo[0], lo[1], lo[2]), v3(hi[0], hi[1], hi[2]), u);
                if (internal) {
                    child = w1.x + meta;
                } else if (inst != kInvalid) {
                    tri = hit;
                } else if (hit) {  // an instance: its object's own bounds, as trace_step
                    inst = __ldg(items + w1.y + (meta & 31u));
                    const DevInstance* I = S.insts + inst;
                    const float4 l = __ldg(&I->olo), h = __ldg(&I->ohi);
                    const Beam ob = make_beam(tb, I->inv);
                    float u2;
                    const V3 err = v3(1e-6f * (fabsf(l.x) + fabsf(h.x)), 1e-6f * (fabsf(l.y) + fabsf(h.y)),
                                      1e-6f * (fabsf(l.z) + fabsf(h.z)));
                    hit = beam_meets(ob, v3(l.x, l.y, l.z) - err, v3(h.x, h.y, h.z) + err, u2);
                    u = fmaxf(u, u2);
                    child = __ldg(&I->blas_root);
                }
            }
        }
        const uint32_t hits = __ballot_sync(0xFFFFFFFFu, hit), tris = __ballot_sync(0xFFFFFFFFu, tri);
        __syncwarp();
        // the entries in turn: replaced by their children, or done
        const int groups = min(4, __popc(open));
        uint32_t left = open;
        uint32_t dead = 0;
        for (int k = 0; k < groups; ++k) {
            const int slot = __ffs(left) - 1;
            left &= left - 1u;
            const uint32_t h8 = (hits >> (8 * k)) & 0xFFu, t8 = (tris >> (8 * k)) & 0xFFu;
            const int cnt = __popc(h8);
            if (t8 || n + cnt - 1 > kTileNodes) {
                if (lane == 0) E[slot].done = 1u;
            } else if (cnt == 0) {
                dead |= 1u << slot;
            } else {
                if (g == k && hit) {
                    const int r = __popc(h8 & ((1u << sub) - 1u));
                    E[r == 0 ? slot : n + r - 1] = TileEntry{inst, child, u, 0u};
                }
                n += cnt - 1;
            }
        }
        __syncwarp();
        if (dead) {  // compact
            const TileEntry e = lane < n ? E[lane] : TileEntry{0u, 0u, 0.0f, 0u};
            const bool keep = lane < n && !((dead >> lane) & 1u);
            const uint32_t km = __ballot_sync(0xFFFFFFFFu, keep);
            if (keep) E[__popc(km & ((1u << lane) - 1u))] = e;
            n = __popc(km);
            __syncwarp();
        }
    }
    // runs by instance, near first
    const TileEntry e = lane < n ? E[lane] : TileEntry{0xFFFFFFFEu, 0u, kFltMax, 0u};
    float run_u = e.u;
    int same_before = 0, rank_in_run = 0;
    for (int j = 0; j < n; ++j) {
        const uint32_t inst = __shfl_sync(0xFFFFFFFFu, e.inst, j);
        const float u = __shfl_sync(0xFFFFFFFFu, e.u, j);
        if (inst == e.inst) {
            run_u = fminf(run_u, u);
            if (j < lane) ++same_before;
            if (u < e.u || (u == e.u && j < lane)) ++rank_in_run;
        }
    }
    const uint32_t heads = __ballot_sync(0xFFFFFFFFu, lane < n && same_before == 0);
    const int runs = __popc(heads);
    if (runs > kTileRuns) {
        if (lane == 0) {
            out->num_runs = 1u;
            out->run[0] = TileList::Run{kInvalid, 0u, 1u, 0.0f};
            out->node[0] = TileList::Node{root, 0.0f};
        }
        return;
    }
    int run_rank = 0, first = 0, count = 0;
    for (int j = 0; j < n; ++j) {
        const uint32_t inst = __shfl_sync(0xFFFFFFFFu, e.inst, j);
        const float u = __shfl_sync(0xFFFFFFFFu, run_u, j);
        const bool nearer = u < run_u || (u == run_u && inst < e.inst);
        if (inst == e.inst) {
            ++count;
        } else if (nearer) {
            ++first;
            if ((heads >> j) & 1u) ++run_rank;
        }
    }
    if (lane < n) {
        if (same_before == 0)
            out->run[run_rank] = TileList::Run{e.inst, (uint32_t)first, (uint32_t)count, beam ? run_u * tb.cmin : 0.0f};
        out->node[first + rank_in_run] = TileList::Node{e.node, beam ? e.u * tb.cmin : 0.0f};
    }
    if (lane == 0) out->num_runs = (uint32_t)runs;
}

}  // namespace omv
