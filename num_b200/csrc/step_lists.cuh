// step_lists.cuh -- the grids of a step's kernels over the engine's tile lists,
// and the room of those lists (plain C++, also for a host compiler).
//
// A step's graph is kept while lists change, so its grids cover more tiles than
// a list holds: the next power of two.  A list has room for as many entries, so
// that a CTA past the list's end may load its entry together with the list's
// length and drop it.
#pragma once

#include <algorithm>
#include <cstdint>

namespace nm {

// One CTA per tile: the tile count rounded up to a power of two.
inline int tile_bucket(int64_t tiles) {
    int64_t b = 1;
    while (b < tiles) b <<= 1;
    return int(std::min<int64_t>(b, INT32_MAX));
}

// The same for the tiles of systems in diagonal form, 0 without any: what
// bs_spmv_dia's launch follows.
inline int dia_bucket(int64_t tiles) { return tiles > 0 ? tile_bucket(tiles) : 0; }

// bs_spmv_dia's CTAs per tile, as a power of two: enough of them for the GPU,
// from two (2,048 rows each) to one per row block.  The grid does not tell
// which it was (64 tiles by 8 CTAs, 128 by 4 and 256 by 2 are all 512); the
// bucket tells both.
inline int dia_split(int64_t tiles) {
    int split = 1;
    while (split < 4 && (int64_t(tile_bucket(tiles)) << split) < 512) ++split;
    return split;
}

inline int dia_grid(int64_t tiles) { return dia_bucket(tiles) << dia_split(tiles); }

// Entries of a tile list made for up to `tiles` tiles: as many as the grids
// above reach.
inline int64_t tile_list_room(int64_t tiles) {
    return std::max<int64_t>(tiles, tile_bucket(tiles));
}

}  // namespace nm
