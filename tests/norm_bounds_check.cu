// Host-side walk of the addresses that norm_solve (norm_wave.cuh) forms with its helper functions.
#include <cstdio>

#include "norm_wave.cuh"

// The row above: loads of `cols` values every step from the run's first one until its window closes (up to 31 steps
// and a chunk after the last block).
static int row_walk(int nsteps, int cols)
{
    const int values = nsteps * cols;
    int at = 0;
    for (int q = -100; q < nsteps + 31 + 2 * sigk::kNormChunk; ++q) {
        if (at < 0 || at + cols > values) return 1;                           // outside the row
        if (q >= 0 && q < nsteps && at != q * cols) return 2;                 // not the step's block
        at += sigk::norm_row_move(q, nsteps, cols);
    }
    return 0;
}

// A step's rows in a tile whose coarse columns take several steps (orders 3 and up): inside the tile, at the column.
static int tile_walk(long long nc, int order, int cols)
{
    const long long pitch = (nc + 2) / 2 * 2, nref = nc << order;
    const int nsteps = (int)((nref + cols - 1) / cols);
    const long long per_col = (1ll << order) / cols; // steps a column
    for (int q = -100; q < nsteps + 100; q += q > 200 && q < nsteps - 400 ? 397 : 1) {
        const long long at = sigk::norm_col_offset(q, nsteps, cols, order, (int)pitch);
        if (at != (q < 0 || q >= nsteps ? 0 : q / per_col) * pitch) return 1;
    }
    return 0;
}

int main()
{
    for (int order : {3, 4, 6})
        for (long long nc : {1, 2, 33, 500, 40000, 46340, 46342, 50000, 70001})
            if (tile_walk(nc, order, 4)) {
                printf("tile: wrong offset at %lld coarse columns, order %d\n", nc, order);
                return 1;
            }
    for (int cols = 2; cols <= 4; cols += 2)
        for (int nsteps : {1, 2, 3, 16, 17, 33, 1099, 16384})
            if (int bad = row_walk(nsteps, cols)) {
                printf("row above: %s at nsteps = %d, cols = %d\n", bad == 1 ? "read outside the row" : "wrong block",
                       nsteps, cols);
                return 1;
            }
    printf("ok\n");
    return 0;
}
