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

// Columns of 2048 and 4096 points that few blocks work on take the Stockham stages, a column's 256
// or 512 threads on one stage after the other, instead of the in-place columns: the transforms
// while there are at most 3072 points per SM, the multiply of columns without padding while there
// is at most one per SM.  Torque, in place and with these: 2x1024x32 cells 53.6 and 45.5 us, 4x1024x32
// (396 columns) 60.2 and 62.7; 2x2048x16 56.7 and 49.0, 2x2048x32 (198) 65.9 and 69.8; periodic
// 4096x64 82.4 and 68.1, 4096x256 137.7 and 164.5.
inline bool line_columns(int L, long long cols) { return (L == 2048 || L == 4096) && cols * L <= SMS * 3072LL; }
inline bool line_multiply(int L, long long cols) { return (L == 2048 || L == 4096) && cols <= SMS; }

// Columns per block of the parity-split multiply of 2048-point columns: 4, or 2 by the same rule
// (1024 rows of 64 cells 155 -> 126 us a step, of 256 cells 214 -> 186; of 512 cells, 257 blocks
// of 2: 257 -> 305).
inline int split_columns(int ncols, int nsim) { return (long long)((ncols + 1) / 2) * nsim <= SMS ? 2 : 4; }

// Columns per block of the four-step multiply (colmul4_kernel), as a shift of its default 64 / P2
// (P2 threads per column): the default, on grids of columns of up to 128 points as much narrower
// (an eighth at most) as leaves one block per SM; then half or double that (tile -1, +1).  A film
// of 128x32 cells has 129 columns, 17 blocks of the default 8.  Longer columns keep their tile:
// 48-thread blocks of one 256-point column take 11.1 us, 192-thread ones 10.0.  (Within the narrowed
// ones it matters little: films of 32 rows 8.6 us and of 64 rows 10.6 us at -1, 0 and +1.)
inline int colmul4_shift(int L, int P2, long long cols, int tile) {
    int shift = 0;
    while (L <= 128 && shift > -3 && cols < (long long)SMS * (64 / P2 >> -shift)) shift--;
    return std::max(-3, std::min(1, shift + tile));
}

// Rows and threads per block of the four-step row-shaped passes (C2R + epilogue, stage combine;
// rhs.cu).  A full tile (flex = false) is `full` rows of `row_threads` threads each, a
// compile-time constant of the kernel.  A flex launch passes its own rows and may have more
// threads than the row transforms use: the extra ones work on the cells only.
//  * Grids that fill the GPU with full tiles: the full tile, or half of it (tile -1).
//    (1024 rows of 1024 cells, 256 full tiles: in finer ones the torque took 279 us, not 264;
//    both would be 70 less with the columns of today.)
//  * Fewer full tiles than SMs: the block's cells, not bandwidth, set the time (a
//    192-thread block of 8 rows of 128 cells walks 5 cells per thread, one dependent
//    round trip after the other), so the rows spread over up to two blocks per SM with a
//    thread per cell (at most 384), at least 128 cells to a block while that leaves one
//    block per SM.  tile -1: half as many rows.  RK45 step, before and after: 128x128 disk
//    under Slonczewski torque 268 -> 148 us, 128x32 film 154 -> 107, 512x128 strip 214 -> 157.
//  * But never more blocks than the SMs hold at once (fit: the threads that a kernel's registers
//    leave an SM), or a few blocks run alone at the end: RK23 step of 512 rows of 1024 cells, 512
//    blocks at one per SM 339 us, 128 blocks 259; 512 rows of 256 cells 111 -> 96 us, nine
//    simulations of 128x128 cells 118 -> 89.
// The row count changes the block decomposition only; every cell's arithmetic is the same.
struct RowTile {
    bool flex;
    int rpb, threads;
};
inline RowTile row_tile(int full, int row_threads, int nrows, int n2, int nsim, int tile, int fit) {
    auto up32 = [](long long v) { return (int)((v + 31) / 32 * 32); };
    auto blocks = [&](long long rpb) { return (nrows + rpb - 1) / rpb * nsim; };
    const long long rows = (long long)nrows * nsim;
    if (blocks(full) >= SMS) {
        if (tile < 0 && full >= 2 && (full / 2) * row_threads >= 32)
            return {true, full / 2, up32((full / 2) * row_threads)};
        return {false, full, up32(full * row_threads)};
    }
    long long rpb = std::max(rows / (2 * SMS), std::min<long long>((127 + n2) / n2, rows / SMS));
    if (tile < 0) rpb /= 2;
    rpb = std::min<long long>(std::max<long long>(rpb, 1), full);
    for (;; rpb++) {
        const long long cells = rpb * n2, turns = (cells + 383) / 384;
        const int threads = std::max(up32((cells + turns - 1) / turns), up32(rpb * row_threads));
        if (rpb == full || tile < 0 || blocks(rpb) <= (long long)SMS * std::max(1, fit / threads))
            return {true, (int)rpb, threads};
    }
}

// Which kernel sums a convolution's weight gradient, for `stages` of 64 positions and `tiles` of
// 32 x 32 channels: the ring of positions, or the one that stages each tap.  The ring takes 7 us
// however small the sum (its halo, one stage after the other, 9216 reductions a block); the
// other's time grows with stages x (tiles + 3).  32x32 channels, the other and the ring: 4.4 and
// 7.3 us (5 stages), 7.0 and 7.5 (162), 11.0 and 8.4 (324); 64x128, 81 stages: 9.6 and 9.3;
// 256x256, 9: 8.7 and 8.5.
inline bool wgrad_by_ring(long long stages, int tiles) { return stages * (tiles + 3) > 656; }

}  // namespace mm
