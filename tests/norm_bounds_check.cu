// Host-side walk of the addresses that norm_solve (norm_wave.cuh) forms with its helper functions.
#include <cstdio>

#include "norm_wave.cuh"

// The row above, as lane 0 of a warp reads it: loads of `cols` values every step from the run's first one until its
// window closes (up to 31 steps and a chunk after the last block), the pointer moving on at each of the row's steps.
// The warps' rows follow `cols` ones; the first warp of a later group of bands reads the last warp's row.
static int row_walk(int nbands, int nw, int nsteps, int cols)
{
    const int values = sigk::norm_bnd_values(nbands, nw, nsteps, cols);
    for (int band = 1; band < nbands; ++band) {
        const int w = band % nw, row = cols + (w == 0 ? nw - 1 : w - 1) * nsteps * cols;
        int at = row;
        for (int q = -100; q < nsteps + 31 + 2 * sigk::kNormChunk; ++q) {
            if (at < 0 || at + cols > values) return 1;                  // outside the CTA's rows
            if (q >= 0 && q < nsteps && at != row + q * cols) return 2;  // not the step's block
            at += q >= 0 && q < nsteps ? cols : 0;
        }
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
        for (int nw : {1, 2, 8, 16})
            for (int nbands = nw; nbands <= 3 * nw; ++nbands)
                for (int nsteps : {1, 2, 33, 1099})
                    if (int bad = row_walk(nbands, nw, nsteps, cols)) {
                        printf("row above: %s at %d bands, %d warps, nsteps = %d, cols = %d\n",
                               bad == 1 ? "read outside the rows" : "wrong block", nbands, nw, nsteps, cols);
                        return 1;
                    }
    printf("ok\n");
    return 0;
}
