// tiles.h -- rules that choose tiles and kernels by the sizes of a launch.  Plain C++ on the host, so that
// they can be checked without a GPU.
#pragma once
#include <algorithm>
#include <cstddef>

namespace mm {

constexpr int SMS = 148;

// Columns and threads per block of the in-place column passes (colmix.cu), for a column of
// line_bytes in shared memory and `outer` tiles of ncols columns.
//  * 16 columns (128-byte rows) while they fit 50 KB, 4 at least while they fit 200 KB, and
//    fewer, down to 4, for grids of less than one block per SM.
//  * Then half as many while the doubled grid is still at most one block per SM: the block's own
//    time, not its row width, is the pass (RK23 step of 1000 rows of 64 cells: 17 blocks of 4
//    columns 241 us, 65 of one 124; of 256 cells: 65 blocks 287, 129 194, 257 221).  Short lines
//    (less than 16 KB a block) keep 4.
//  * 512 threads where a block has an SM to itself, by the grid or by its shared memory, else 256
//    (1000 rows of 1024 cells, 4 columns in 192 KB: 746 -> 636 us; 600 rows, two blocks of 115 KB
//    per SM: 415 with 256 threads, 432 with 512).
struct ColTile {
    int tc, threads;
};
inline ColTile col_tiles(size_t line_bytes, int ncols, long long outer) {
    auto blocks = [&](int tc) { return (ncols + tc - 1) / tc * outer; };
    int tc = 16;
    while (tc > 4 && line_bytes * tc > 50 * 1024) tc /= 2;
    while (tc > 2 && line_bytes * tc > 200 * 1024) tc /= 2;
    while (tc > 4 && blocks(tc) < SMS) tc /= 2;
    while (tc > 1 && line_bytes * tc >= 16 * 1024 && blocks(tc / 2) <= SMS) tc /= 2;
    const bool alone = blocks(tc) <= SMS || 2 * (line_bytes * tc + 1024) > 228 * 1024;
    return {tc, alone ? 512 : 256};
}

// Columns per block of the parity-split multiply of 2048-point columns: 4, or 2 by the same rule
// (1024 rows of 64 cells 155 -> 126 us a step, of 256 cells 214 -> 186; of 512 cells, 257 blocks
// of 2: 257 -> 305).
inline int split_columns(int ncols, int nsim) { return (long long)((ncols + 1) / 2) * nsim <= SMS ? 2 : 4; }

// Which kernel sums a convolution's weight gradient, for `stages` of 64 positions and `tiles` of
// 32 x 32 channels: the ring of positions, or the one that stages each tap.  The ring takes 7 us
// however small the sum (its halo, one stage after the other, 9216 reductions a block); the
// other's time grows with stages x (tiles + 3).  32x32 channels, the other and the ring: 4.4 and
// 7.3 us (5 stages), 7.0 and 7.5 (162), 11.0 and 8.4 (324); 64x128, 81 stages: 9.6 and 9.3;
// 256x256, 9: 8.7 and 8.5.
inline bool wgrad_by_ring(long long stages, int tiles) { return stages * (tiles + 3) > 656; }

}  // namespace mm
