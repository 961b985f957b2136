// How a split-K launch divides a session's tiles among its splits: plain arithmetic for host and device (tests/test_split_bounds_cpu.py runs it).
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define B200KV_HD __host__ __device__ __forceinline__
#else
#define B200KV_HD inline
#endif

namespace b200kv {

// The first of `total` tiles that belongs to part `i` of `parts` (i <= parts <= kMaxSplitsPerSession): floor(total * i / parts), a product that
// does not fit 32 bits, from 32-bit divisions.
B200KV_HD uint32_t part_begin(uint32_t total, uint32_t i, uint32_t parts) {
    const uint32_t q = total / parts, r = total - q * parts;
    return q * i + r * i / parts;
}

// Splits of one session for a pipelined kernel whose CTAs walk whole tiles, by the least estimated time (nanoseconds, fitted by the kernels that call this): the
// longest split's tiles, the first three of which may cost less (they are on their way before the launch may begin), every split's partial on its way
// through the merge, and splits past `on_time`, whose CTAs find a place only when the launch before has left its own.  Looked at are the fewest splits for every
// longest part from the shortest possible to eight tiles more.  Parts of `fill` tiles or more share the memory's bandwidth: then as many of one length as there are places.
struct SplitCosts { uint32_t early_tile, tile, split, late, per_late, fill; };
B200KV_HD uint32_t cheapest_splits(uint32_t tiles, uint32_t most, uint32_t on_time, SplitCosts c) {
    if (tiles == 0 || most <= 1) return 1;
    const uint32_t shortest = (tiles + most - 1) / most;
    uint32_t best = 1, best_longest = tiles;
    uint64_t least = ~0ull;
    for (uint32_t longest = shortest; longest <= tiles && longest <= shortest + 8; ++longest) {
        const uint32_t splits = (tiles + longest - 1) / longest, early = longest < 3 ? longest : 3;
        const uint64_t cost = static_cast<uint64_t>(early) * c.early_tile + static_cast<uint64_t>(longest - early) * c.tile + static_cast<uint64_t>(splits) * c.split +
                              (splits > on_time ? c.late + static_cast<uint64_t>(splits - on_time) * c.per_late : 0);
        if (cost < least) { least = cost; best = splits; best_longest = longest; }
    }
    if (best_longest >= c.fill && best_longest > 1) {
        const uint32_t same = (tiles - 1) / (best_longest - 1), room = best <= on_time && on_time < most ? on_time : most;   // the most parts of that length
        best = same < room ? same : room;
    }
    return best;
}

// Splits per kv head whose CTAs find an SM only when the mergers of the launch before leave theirs, one CTA per SM.  Only under launch overlap, behind a
// launch of the same shape that merges inside (`mergers` units per kv head) and where both together are more than the device holds; never half of
// the splits or more.
B200KV_HD uint32_t late_splits(bool overlap, bool merge_inside, uint32_t kv_heads, uint32_t num_splits, uint32_t mergers, uint32_t sms) {
    if (!overlap || !merge_inside) return 0;
    const uint32_t ctas = kv_heads * (num_splits + (mergers < num_splits ? mergers : num_splits));
    const uint32_t late = ctas > sms ? (ctas - sms + kv_heads - 1) / kv_heads : 0;
    return 2 * late < num_splits ? late : 0;
}

// Tiles [begin, end) of split `i` of `splits` of one session, for CTAs of WARPS warps; a round is one tile per warp.  Even parts (part_begin), or the last
// `late` parts WARPS tiles shorter than the others: only where that leaves the longest part its number of rounds and the last one a round less, and from
// three rounds on.  Written for few instructions: it stands at the start of a launch that is a chain of latencies.
struct TileRange { uint32_t begin, end; };
template <uint32_t WARPS>
B200KV_HD TileRange split_tiles(uint32_t tiles, uint32_t i, uint32_t splits, uint32_t late) {
    uint32_t q = tiles / splits, r = tiles - q * splits;
    if (late != 0) {
        const uint32_t rounds = (q + (r != 0) + WARPS - 1) / WARPS;   // of the longest even part
        if (rounds >= 3 && tiles + late * WARPS <= rounds * WARPS * splits)
            for (r += late * WARPS; r >= splits; r -= splits) ++q;    // parts of the tiles and what the late ones fall short of
        else late = 0;
    }
    const uint32_t extra = r * i / splits, next = r * i - extra * splits + r;
    const uint32_t cut = i + late > splits ? (i + late - splits) * WARPS : 0u, begin = q * i + extra - cut;
    return {begin, begin + q + (next >= splits) - (i + late >= splits ? WARPS : 0u)};
}

}  // namespace b200kv
