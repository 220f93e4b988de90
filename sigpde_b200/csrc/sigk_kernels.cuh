// sigk_kernels.cuh -- persistent-warp kernels built on warp_solve (wave.cuh).
//
//   pair_kernel       pairwise / Gram / symmetric-Gram signature kernels
//
// A grid of 4-warp blocks sized to the resident capacity of the device; warp w
// handles work items w, w + W, w + 2W, ... (W = warps in the grid).  Gram items
// are numbered row-major, so neighbouring warps share x_i and read neighbouring
// y_j (L1/L2 reuse).
#pragma once

#include <type_traits>

#include "wave.cuh"

namespace sigk {

enum : int { kOpPairwise = 0, kOpGram = 1, kOpGramSym = 2 };

constexpr int kWarpsPerBlock = 4;

struct PairParams {
    int op;
    const void *x;
    const void *y;
    int64_t nx, ny;     // path counts (pairwise: batch in both)
    int64_t ncx, ncy;   // coarse cells per side (len - 1)
    int64_t d;
    int order;
    double fscale;      // static_scale * 4^-order (path mode) or 1 (increment mode)
    const void *sx;
    const void *sy;
    const void *dx;     // path mode: scaled differences (nx, d, ncx) in T, dimension-major (delta_kernel)
    const void *dy;     // (ny, d, ncy)
    const void *inc;    // increment mode only
    int64_t is0, is1, is2, is3;
    // matrix mode (tensor-core increments, tc.cuh): pair (xi, yj)'s increments start at
    // mat + yj * ncy * mat_ld + (xi - x0) * mat_rows_x (Gram ops; pairwise: mat + (item - item0) * ncy *
    // mat_rows_x), mat_ld (pairwise: mat_rows_x) floats per coarse column
    const void *mat;         // float (tensor-core increments) or double (dgemm_inc_kernel) elements
    const unsigned *mat_err; // non-zero: the GEMM gave up a wait, the matrix is incomplete (results NaN)
    int64_t mat_ld, mat_rows_x, x0;
    int64_t item0;      // first item of this launch (matrix mode works in chunks of x paths)
    void *out;
    int64_t out_ld;
    int64_t nitems;
    void *bnd;          // per-warp boundary rows (multi-band pairs only)
    int64_t bnd_stride; // elements per warp
    int stage_smem;     // 1: dx rows staged in shared memory
};

// Lower-triangle index w -> (i, j), i >= j, w = i*(i+1)/2 + j.
__device__ __forceinline__ void tri_decode(int64_t w, int64_t &i, int64_t &j)
{
    int64_t r = (int64_t)((sqrt(8.0 * (double)w + 1.0) - 1.0) * 0.5);
    while (r * (r + 1) / 2 > w) --r;
    while ((r + 1) * (r + 2) / 2 <= w) ++r;
    i = r;
    j = w - r * (r + 1) / 2;
}

template <typename TIN>
__device__ __forceinline__ double scale_at(const void *s, int64_t i)
{
    return s ? (double)reinterpret_cast<const TIN *>(s)[i] : 1.0;
}

enum : int { kPairDelta = 0, kPairGiven = 1, kPairMat = 2, kPairMat64 = 3 };

template <typename T, typename TIN, int R, int O, int MODE>
__global__ void __launch_bounds__(kWarpsPerBlock * 32) pair_kernel(PairParams p)
{
    using BS = BlockShape<R, O>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const int64_t gwarp = (int64_t)blockIdx.x * kWarpsPerBlock + wib;
    const int64_t nwarps = (int64_t)gridDim.x * kWarpsPerBlock;
    const SolveGeom g = make_geom<R, O>(p.ncx, p.ncy, p.order);
    T *bnd = p.bnd ? reinterpret_cast<T *>(p.bnd) + gwarp * p.bnd_stride : nullptr;
    TIN *out = reinterpret_cast<TIN *>(p.out);

    for (int64_t item0 = gwarp; item0 < p.nitems; item0 += nwarps) {
        const int64_t item = p.item0 + item0;
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
        double s = p.fscale;
        if (p.sx) s *= scale_at<TIN>(p.sx, xi);
        if (p.sy) s *= scale_at<TIN>(p.sy, yj);

        T val;
        if constexpr (MODE == kPairMat || MODE == kPairMat64) {
            using TM = typename std::conditional<MODE == kPairMat64, double, float>::type;
            MatIncs<T, BS::RC, TM> src;
            const TM *mat = reinterpret_cast<const TM *>(p.mat);
            if (p.op == kOpPairwise) {
                src.base = mat + (item - p.item0) * p.ncy * p.mat_rows_x;
                src.ld = p.mat_rows_x;
            } else {
                src.base = mat + yj * p.ncy * p.mat_ld + (xi - p.x0) * p.mat_rows_x;
                src.ld = p.mat_ld;
            }
            src.ncy = p.ncy;
            val = (p.mat_err == nullptr || *p.mat_err == 0) ? warp_solve<T, R, O>(g, src, bnd) : T(NAN);
        } else if constexpr (MODE == kPairGiven) {
            GivenIncs<T, TIN, BS::RC> src;
            const TIN *base = reinterpret_cast<const TIN *>(p.inc);
            if (p.op == kOpPairwise) {
                src.inc = base + item * p.is0;
                src.si = p.is1;
                src.sj = p.is2;
            } else {
                src.inc = base + xi * p.is0 + yj * p.is1;
                src.si = p.is2;
                src.sj = p.is3;
            }
            src.fscale = T(s);
            val = warp_solve<T, R, O>(g, src, bnd);
        } else {
            DeltaIncs<T, BS::RC> src;
            src.dX = reinterpret_cast<const T *>(p.dx) + xi * p.d * p.ncx;
            src.dY = reinterpret_cast<const T *>(p.dy) + yj * p.d * p.ncy;
            src.d = p.d;
            src.ncy = p.ncy;
            src.dxs = p.stage_smem ? reinterpret_cast<T *>(smem_raw) + (int64_t)wib * BS::RC * p.d * 32 : nullptr;
            val = warp_solve<T, R, O>(g, src, bnd);
        }
        if (lane == 0) {
            if (p.op == kOpPairwise) {
                out[item] = TIN(val);
            } else {
                out[xi * p.out_ld + yj] = TIN(val);
                if (p.op == kOpGramSym && xi != yj) out[yj * p.out_ld + xi] = TIN(val);
            }
        }
    }
}

} // namespace sigk
