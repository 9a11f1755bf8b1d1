// Sizes of the wavefront renderer's scratch memory: the arrays of one wave, and
// where in them the light subpaths' queues lie while they run beside the camera
// rays.  Host code without CUDA headers, so that it can be checked on its own.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace omv {

constexpr int kMaxCounters = 512;

// Waves of at most this many paths run their light subpaths beside the camera
// rays (64x64x1 401 -> 382 us, 256x256x16 997 -> 955); larger ones keep the GPU
// busy by themselves, and the queues' 80 bytes per path are better spent on
// fewer waves.
constexpr int64_t kBesideLightPaths = 1 << 22;

// Entries of the ray queues and of the hits of a scratch for waves of up to
// `wave_cap` paths.  With `beside`, every wave that it takes and that runs its
// light subpaths beside the camera rays finds a second set of `wave` entries
// behind the first.
inline int64_t queue_entries(int64_t wave_cap, bool beside)
{
    return beside ? std::max(wave_cap, std::min(2 * wave_cap, 2 * kBesideLightPaths)) : wave_cap;
}

// First entry of the light subpaths' queues of a wave of `wave` paths in arrays
// of `queue_cap` entries; 0: no room for queues of their own (or too large a
// wave), the subpaths run before the camera rays in the same entries.
inline int64_t light_queue_first(int64_t wave, int64_t queue_cap)
{
    return wave <= kBesideLightPaths && wave <= queue_cap / 2 ? queue_cap - wave : 0;
}

// Byte offsets of one wave's arrays inside a single scratch block (each array
// starts on a 256-byte boundary).
struct ScratchLayout {
    size_t tp, rad, ltp, lrad, lmeta, lvp, lvr, rq0, rq1, hits, pjob, sq, ctr, stats, tiles, bytes;
};

// tile_bytes: room for the tile lists of a frame of several waves
inline ScratchLayout scratch_layout(int64_t wave_cap, int64_t queue_cap, int light_slots, int shadow_slots,
                                    size_t tile_bytes = 0)
{
    const size_t W = (size_t)wave_cap, Q = (size_t)queue_cap;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        size_t o = off;
        off += (bytes + 255) & ~(size_t)255;
        return o;
    };
    ScratchLayout L;
    L.tp = take(W * 16);
    L.rad = take(W * 16);
    L.ltp = take(W * 16);
    L.lrad = take(W * 16);
    L.lmeta = take(W * 4);
    L.lvp = take((size_t)light_slots * W * 16);
    L.lvr = take((size_t)light_slots * W * 16);
    L.rq0 = take(Q * 32);
    L.rq1 = take(Q * 32);
    L.hits = take(Q * 16);
    L.pjob = take(W * 4);
    L.sq = take((size_t)shadow_slots * W * 48 + 48);
    L.ctr = take(kMaxCounters * 4);
    L.stats = take(16 * 8);
    L.tiles = take(tile_bytes);
    L.bytes = off;
    return L;
}

// Scratch bytes of one path: tp rad ltp lrad (16 B each), lmeta 4, light
// vertices 32 per slot, two ray-queue entries 64, hit 16, batch job 4, shadow
// entries 48 per slot (each array is further rounded up to 256 bytes).
inline size_t path_scratch_bytes(int light_slots, int shadow_slots)
{
    return 68 + 32 * (size_t)light_slots + 84 + 48 * (size_t)shadow_slots;
}

}  // namespace omv
