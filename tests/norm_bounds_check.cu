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

int main()
{
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
