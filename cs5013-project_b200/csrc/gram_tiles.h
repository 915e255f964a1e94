// gram_tiles.h -- the order in which a CTA of the tensor-core prune goes through the tiles
// of its candidates' Gram matrix, and where it stops.  Plain C++, no device types.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define VANN_TILES_FN __device__ __forceinline__
#else
#define VANN_TILES_FN inline
#endif

namespace vann {

// Tiles of 128 rows x COLS columns on and below the diagonal of an m x m matrix, row block
// by row block; the caller has issued the first one (0, 0).
//   row(r)       before the tiles of row block r
//   issue(r, c)  starts every other tile; the accumulator is free by then
//   wait()       the tile has arrived, or false: this thread gave up waiting
//   read(r, c)   takes the tile
//   stop(late)   a barrier of the CTA: whether any thread's wait gave up (late: this one's)
// False when a wait gave up: no tile is issued or waited for after that one, so giving up
// takes the bound of one wait and not of one per tile.
template <uint32_t COLS, typename Row, typename Issue, typename Wait, typename Read, typename Stop>
VANN_TILES_FN bool gram_tiles(uint32_t m, Row row, Issue issue, Wait wait, Read read, Stop stop) {
    bool late = false;
    for (uint32_t r = 0; 128u * r < m; ++r) {
        row(r);
        const uint32_t ncols = m < 128u * (r + 1u) ? m : 128u * (r + 1u);
        for (uint32_t c = 0; COLS * c < ncols; ++c) {
            if (r != 0u || c != 0u) {
                if (stop(late)) return false;
                issue(r, c);
            }
            late |= !wait();
            read(r, c);
        }
    }
    return !stop(late);
}

}  // namespace vann
