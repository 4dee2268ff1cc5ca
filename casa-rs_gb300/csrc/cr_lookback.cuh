// cr_lookback.cuh -- the running count before a tile, from the earlier tiles'
// published words (Merrill and Garland's decoupled look-back).
//
// A tile's word is 0 until published, then kind << 32 | count: kind 1 the
// tile's own count, kind 2 the count up to and including the tile.  Tiles take
// their numbers from a ticket counter, so every tile waited for has started;
// each wait is bounded all the same.
#pragma once

#include "cr_internal.cuh"

namespace cr {

// Called by one whole warp with the tile's own count; returns the count of
// all earlier tiles, or sets *good to false when a wait gave up.
__device__ __forceinline__ uint32_t tile_lookback(unsigned long long* state, int64_t tile,
                                                  uint32_t count, bool* good) {
    const int lane = threadIdx.x & 31;
    volatile unsigned long long* st = state;
    if (lane == 0 && tile > 0) st[tile] = 1ull << 32 | count;
    uint32_t before = 0;
    bool ok = true;
    for (int64_t p = tile - 1 - lane;; p -= 32) {
        // 32 predecessors at a time, lane 0 the nearest; before tile 0 lies 0
        unsigned long long w = p >= 0 ? st[p] : 2ull << 32;
        for (long long polls = 0; (w >> 32) == 0;) {
            if (++polls > kLookbackPolls) {
                ok = false;
                break;
            }
            w = st[p];
        }
        const unsigned full = __ballot_sync(0xffffffffu, (w >> 32) == 2);
        const int stop = full ? __ffs(full) - 1 : 31;
        before += __reduce_add_sync(0xffffffffu, lane <= stop ? (uint32_t)w : 0u);
        ok = __all_sync(0xffffffffu, ok);
        if (full || !ok) break;
    }
    // a tile whose wait gave up publishes no total, so every later tile gives up too
    if (lane == 0 && ok) st[tile] = 2ull << 32 | (before + count);
    *good = ok;
    return before;
}

}  // namespace cr
