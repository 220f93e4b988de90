// pair_wave.cuh -- few pairs: one CTA solves a pair, in one launch.
//
// The streaming wavefronts give a warp a run of pairs.  A call with no more pairs
// than the device has warps is bound by one pair's latency there, and by the
// launches that write the differences first: a step of a lone warp costs its
// instructions three times over, since nothing else fills their latencies.  Here
// the CTA forms the pair's differences and coarse increments in shared memory
// and solves with one warp per band in lockstep (norm_wave.cuh), whose step loop
// carries no checks.  The differences, the sums and the cells are those of
// delta_kernel and the float64 wavefronts, in the same order: values agree bit
// for bit, so a request's result does not depend on how many pairs it is cut
// into.
#pragma once

#include "norm_wave.cuh"

namespace sigk {

struct PairWaveParams {
    int op;
    int in64;            // points, scales and output are float64
    const void *x, *y;   // (n_x, ncx + 1, d), (n_y, ncy + 1, d)
    const void *sx, *sy; // per-path scales or null
    double f;            // static scale * 4^-order, on the x side
    int64_t ny;
    int nc, ncy;         // coarse rows, columns
    int64_t d;
    int order;
    void *out;
    int64_t out_ld;
    int64_t nitems;
    int nbands, nw, nsteps, pitch, col0;
    int tile;            // values of the increment tile
};

// scaled differences of one path, dst[k * nc + c], as delta_kernel forms them
template <typename TIN>
__device__ __forceinline__ void pair_wave_diffs(const void *x_, const void *s_, int64_t path, int nc, int d, double f,
                                                double *dst)
{
    const TIN *x = reinterpret_cast<const TIN *>(x_) + path * (nc + 1) * d;
    const double g = s_ ? f * (double)reinterpret_cast<const TIN *>(s_)[path] : f;
    for (int e = threadIdx.x; e < nc * d; e += blockDim.x) {
        const int c = e / d, k = e - c * d;
        dst[k * nc + c] = ((double)x[e + d] - (double)x[e]) * g;
    }
}

template <int R, int O>
__global__ void __launch_bounds__(NormShape<R, O>::MAXW * 32, 1) pair_wave_kernel(PairWaveParams p)
{
    using NS = NormShape<R, O>;
    extern __shared__ __align__(16) double pair_smem[];
    __shared__ double s_val;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int ncx = p.nc, ncy = p.ncy, d = (int)p.d;
    double *tile = pair_smem, *bnd = tile + p.tile;
    double *dx = bnd + norm_bnd_values(p.nbands, p.nw, p.nsteps, NS::C), *dy = dx + ncx * d;
    double *cols = tile + p.col0 * p.pitch;
    if (threadIdx.x < NS::C) bnd[threadIdx.x] = 1.0;
    const int pad = p.pitch - ncx; // zeros below a column's rows, and before the first column
    for (int e = threadIdx.x; e < ncy * pad; e += blockDim.x) cols[(e / pad) * p.pitch + ncx + e % pad] = 0.0;
    for (int e = threadIdx.x; e < p.col0 * p.pitch; e += blockDim.x) tile[e] = 0.0;
    for (int64_t item = blockIdx.x; item < p.nitems; item += gridDim.x) {
        int64_t xi, yj;
        if (p.op == kOpPairwise) {
            xi = item;
            yj = item;
        } else if (p.op == kOpGram) {
            xi = item / p.ny;
            yj = item - xi * p.ny;
        } else {
            tri_decode(item, xi, yj);
        }
        if (p.in64) {
            pair_wave_diffs<double>(p.x, p.sx, xi, ncx, d, p.f, dx);
            pair_wave_diffs<double>(p.y, p.sy, yj, ncy, d, 1.0, dy);
        } else {
            pair_wave_diffs<float>(p.x, p.sx, xi, ncx, d, p.f, dx);
            pair_wave_diffs<float>(p.y, p.sy, yj, ncy, d, 1.0, dy);
        }
        __syncthreads();
        for (int cj = w * 8; cj < ncy; cj += warps * 8) { // a warp takes 8 columns, its lanes the rows
            for (int ci = lane; ci < ncx; ci += 32) {
                double acc[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[j] = 0.0;
                for (int k = 0; k < d; ++k) {
                    const double a = dx[k * ncx + ci];
                    const double *row = dy + k * ncy;
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[j] = fma(a, row[cj + j < ncy ? cj + j : cj], acc[j]);
                }
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (cj + j < ncy) cols[(cj + j) * p.pitch + ci] = acc[j];
            }
        }
        __syncthreads();
        if (w < p.nw) {
            const double v = norm_solve<R, O, true, true, false>(p, tile, bnd, 1.0, &s_val);
            if (threadIdx.x == 0) {
                const int64_t at = p.op == kOpPairwise ? item : xi * p.out_ld + yj, to = yj * p.out_ld + xi;
                const bool mirror = p.op == kOpGramSym && xi != yj;
                if (p.in64) {
                    reinterpret_cast<double *>(p.out)[at] = v;
                    if (mirror) reinterpret_cast<double *>(p.out)[to] = v;
                } else {
                    reinterpret_cast<float *>(p.out)[at] = (float)v;
                    if (mirror) reinterpret_cast<float *>(p.out)[to] = (float)v;
                }
            }
        }
        __syncthreads(); // the differences and the tile are free for the next pair
    }
}

} // namespace sigk
