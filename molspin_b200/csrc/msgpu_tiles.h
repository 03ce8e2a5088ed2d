// msgpu_tiles.h -- tile sizes of the streamed kernels and the rows of partial
// sums that they leave: the allocation, the launches and the host tests use the
// same rules.
#pragma once

#include <stddef.h>

#include <algorithm>

namespace msgpu {

// Rows per tile: keep about 64-128 row tiles per trajectory tile so that the
// partial-sum buffers stay small and every SM has several CTAs.
inline int pick_rows_per_tile(int D)
{
    int R = D / 64;
    R = std::max(8, std::min(512, R));
    R = (R + 7) / 8 * 8;
    return R;
}

// complex128 partial sums, in rows of one FP64 value a trajectory: Gram-Schmidt
// leaves m + 1 complex sums a row tile; the three-term recurrence, which leaves
// one real sum a tile, stays below this number.
inline size_t partial_rows_d(int ntiles, int m) { return 2 * static_cast<size_t>(ntiles) * (m + 1); }

// Quartets per CTA of k_lanczos_apply_d: 16, or 8 while 16 leaves under 8 CTAs
// an SM (D = 16384, us per launch: 512 trajectories 176 with 8 or 16, 185 with
// 32, 223 with 64), and as many more as it takes for the tiles to fit max_tiles
// rows of partial sums (a Krylov dimension of a few at a large D).
inline int quartet_tile_d(int Q, int width, size_t max_tiles)
{
    const int tile = static_cast<long long>(Q) / 16 * (width / 32) >= 8 * 148 ? 16 : 8;
    const size_t least = (static_cast<size_t>(Q) + max_tiles - 1) / max_tiles;
    return std::max(tile, static_cast<int>((least + 7) / 8 * 8));
}

}  // namespace msgpu
