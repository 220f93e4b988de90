// norm_wave.cuh -- robust normalisation: the per-path Chandrupatla root-find,
// every bracket iteration re-solving the path's self-kernel on chip.
//
// A call is bound by latency: about ten solves of one path follow one another,
// and a solve's cells lie on n + m anti-diagonals.  So one CTA works on one
// path, with one warp per band of 32 R refined rows, and R is small.  The warps
// run in lockstep: warp w takes the same step kNormLag steps after warp w - 1,
// and a barrier every kNormChunk steps publishes the bands' bottom rows, so no
// warp polls another's progress.  The coarse increments are formed once per
// path, into shared memory where they fit, else into a tile in the workspace
// that stays in the L2.  Measured, before (one warp a path, increments re-formed
// each solve above 48 KB; or bands that poll each other through global memory)
// and now, us a call: 24 paths, L = 220, d = 8, order 1: 4069, 553; 512 paths,
// L = 64, d = 16, order 1: 297, 152; 8 paths, L = 256, d = 32, order 2: 16185,
// 1191; 32 paths, L = 128, d = 32, order 1: 1642, 301.  Calls of many short paths,
// or of long ones in number, take a warp a path instead (norm_warp.cuh).
//
// The increments' sums are those of the other kernels, in the same order; the
// root-find's cells are stencil_chain's, whose roundings differ from theirs.
#pragma once

#include "sigk_kernels.cuh"

namespace sigk {

struct NormParams {
    int64_t n;           // paths
    int nc, order;
    int64_t d;
    const double *dx;    // path differences (n, d, nc), dimension-major, unscaled; null: increments given
    const void *inc;     // given increments, element (b, i, j) at b * is0 + i * is1 + j * is2
    int64_t is0, is1, is2;
    int in64;            // inc and lam are float64
    double fscale;       // static_scale * 4^-order (1: increments given)
    int nbands, nw;      // bands of a path, warps that solve (bands go in groups of nw)
    int nsteps;          // lane steps of a band
    int pitch;           // tile: values a column (its rows, then zeros)
    int col0;            // tile column of coarse column 0 (1: a zero column before it)
    int64_t tile;        // values of a tile
    double *tiles;       // one tile a CTA, where it is not in shared memory
    double *bnd;         // C ones and nw rows a CTA, where they are not in shared memory; norm_warp_kernel: a row a warp
    int64_t bnd_stride;  // norm_warp_kernel: values of a row, and of a warp's shared memory
    int64_t smem_values;
    double *knorm;       // builtin: output (may be null); external: input
    const double *fnorm; // null: builtin f(s) = 2 - 1/(1 + log s)
    double tol;
    int maxit;
    void *lam;
    int *iters;
};

template <int R, int O>
struct NormShape {
    static constexpr int C = O == 0 ? 2 : 4;                                  // columns a step
    static constexpr int RC = O < 4 && (R >> O) > 0 ? (R >> O) : 1;          // coarse rows a lane
    static constexpr int CC = O < 4 && (C >> O) > 0 ? (C >> O) : 1;          // coarse columns a step
    static constexpr bool WHOLE = O < 4 && (C >> O) > 0;                     // steps hold whole coarse columns
    static constexpr int MAXW = R == 16 ? 8 : 16;                            // warps a CTA
    // steps that increments are loaded ahead: from shared memory, and from the L2
    __host__ __device__ static constexpr int ahead(bool smem) { return smem ? 1 : RC * CC <= 4 ? 4 : 2; }
    __host__ __device__ static constexpr int rc_of(int r) { return RC == 1 ? 0 : r >> O; }
    __host__ __device__ static constexpr int cc_of(int c) { return CC == 1 ? 0 : c >> O; }
};

// Memory that a lane addresses every step: shared (32-bit addresses, immediate
// offsets) or global.  Stores are predicated rather than branched around, and
// loads are unconditional: a branch a step for lane 0's row or lane 31's costs
// as much as the step's cells.
template <bool SMEM>
struct NormMem;

template <>
struct NormMem<true> {
    unsigned a;
    __device__ __forceinline__ explicit NormMem(const double *p) : a((unsigned)__cvta_generic_to_shared(p)) {}
    __device__ __forceinline__ void move(int values) { a += values * 8; }
    __device__ __forceinline__ double get(int i) const
    {
        double v;
        asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a + i * 8) : "memory");
        return v;
    }
    __device__ __forceinline__ double2 get2(int i) const
    {
        double2 v;
        asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a + i * 8) : "memory");
        return v;
    }
    __device__ __forceinline__ void put2(int i, double x, double y, bool on) const
    {
        asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %3, 0;\n @p st.shared.v2.f64 [%0], {%1, %2};\n}" ::"r"(a + i * 8),
                     "d"(x), "d"(y), "r"((int)on)
                     : "memory");
    }
};

template <>
struct NormMem<false> {
    const double *a;
    __device__ __forceinline__ explicit NormMem(const double *p) : a(p) {}
    __device__ __forceinline__ void move(int64_t values) { a += values; }
    __device__ __forceinline__ double get(int i) const
    {
        double v;
        asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(a + i) : "memory");
        return v;
    }
    __device__ __forceinline__ double2 get2(int i) const
    {
        double2 v;
        asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(a + i) : "memory");
        return v;
    }
    __device__ __forceinline__ void put2(int i, double x, double y, bool on) const
    {
        asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %3, 0;\n @p st.global.v2.f64 [%0], {%1, %2};\n}" ::"l"(a + i),
                     "d"(x), "d"(y), "r"((int)on)
                     : "memory");
    }
};

constexpr int kNormChunk = 4;              // steps between barriers
constexpr int kNormLag = 32 + kNormChunk;  // a row is read (a step ahead) at least one barrier after it is written

// k(x,x), f(k) and the Chandrupatla iteration for one path, given solve(s) =
// k at increments scaled by s: sigpde/cuda_pairwise_kernels.py:88-165 with
// the argument order of sigpde/torch/kernel.py:186-193: g(l) = k(l x) - f(k),
// g(0) = 1 - f(k), g(1) = k - f(k).  All bracket state is float64 and uniform
// across the threads that call it (solve returns the same value to all of
// them); `writer` stores k(x,x).
template <class Solve>
__device__ __forceinline__ void normalize_path(const NormParams &p, int64_t b, bool writer, Solve &&solve,
                                               double &out, int &it)
{
    double fk = 0.0, a = 0.0, bb = 1.0, c = 0.0, fa = 0.0, fb = 0.0, fc = 0.0, t = 0.5, xt = 1.0;
    bool norm = p.fnorm == nullptr; // the first solve is k(x,x)
    auto start = [&](double k) {    // the bracket [0, 1]; false where there is nothing to search
        fa = 1.0 - fk;
        fb = k - fk;
        fc = fa;
        xt = a + t * (bb - a);
        return k >= 1.0 && p.maxit > 0; // lambda is forced to 0 for k < 1 (kernel.py:195)
    };
    out = 0.0;
    it = 0;
    if (!norm) {
        fk = p.fnorm[b];
        if (!start(p.knorm[b])) return;
    }
    while (true) { // one call of solve in the code: it is inlined
        const double sol = solve(xt * xt);
        if (norm) {
            norm = false;
            const double k = isnan(sol) ? __longlong_as_double(0x7ff0000000000000LL) : sol; // NaN -> +inf (kernel.py:183)
            fk = 2.0 - 1.0 / (1.0 + log(k));                                                // kernel.py:23-24
            if (p.knorm && writer) p.knorm[b] = k;
            if (!start(k)) return;
            continue;
        }
        const double ft = isnan(sol) ? __longlong_as_double(0x7ff0000000000000LL) : sol - fk;
        ++it;
        if (ft * fa >= 0) {
            c = a;
            fc = fa;
        } else {
            c = bb;
            bb = a;
            fc = fb;
            fb = fa;
        }
        a = xt;
        fa = ft;
        if (fabs(fa) < fabs(fb)) {
            out = a;
            if (fabs(fa) < p.tol) return;
        } else {
            out = bb;
            if (fabs(fb) < p.tol) return;
        }
        const double xi = (a - bb) / (c - bb);
        const double phi = (fa - fb) / (fc - fb);
        if (phi * phi < xi && (1 - phi) * (1 - phi) < 1 - xi)
            t = fa / (fb - fa) * fc / (fb - fc) + (c - a) / (bb - a) * fa / (fc - fa) * fb / (fc - fb);
        else
            t = 0.5;
        if (!(0 < t && t < 1)) t = 0.5;
        if (it >= p.maxit) return;
        xt = a + t * (bb - a);
    }
}

// Values of a CTA's boundary rows: `cols` ones (the row above the first band), then the bottom rows of the nw solving
// warps.  Lane 0's pointer to the row above moves on at each of a row's steps, and the loads go on until the warp's
// window of steps closes: where there are several groups of bands, the first warp of a group reads one block past the
// last row.  (A pointer that stays on the last block needs a register more in the step loop, which spills: 24 paths,
// L = 220, d = 8, order 1: 540 us instead of 531.)
__host__ __device__ constexpr int norm_bnd_values(int nbands, int nw, int nsteps, int cols)
{
    return (nbands > 1 ? nw * nsteps + 1 : 1) * cols + (nbands > nw ? cols : 0);
}

// Values from a lane's rows of the first coarse column to those of step q, where a coarse column takes several steps
// (steps outside the run stay on the first one).  A tile in the workspace has nc * pitch values: past 2^31 from about
// 46000 coarse columns on.
__host__ __device__ constexpr int64_t norm_col_offset(int q, int nsteps, int cols, int order, int pitch)
{
    return (int64_t)((((unsigned)q < (unsigned)nsteps ? q : 0) * cols) >> order) * pitch;
}

// of the solving warps
__device__ __forceinline__ void norm_barrier(int warps)
{
    if (warps > 1)
        asm volatile("bar.sync 1, %0;" ::"r"(warps * 32) : "memory");
    else
        __syncwarp();
}

// The path's coarse increments by the whole CTA: (ci, cj) at tile[(cj + col0) *
// pitch + ci], zeros below a column's rows and in column 0 where col0 = 1.  A
// lane reads its rows of a column without a bound check: lanes beyond the path's
// rows read the zeros.  (In the workspace a layout that holds a warp's step side
// by side, one line a step instead of one a lane, measured no faster.)
__device__ __forceinline__ void norm_build_tile(const NormParams &p, int64_t b, double *tile)
{
    const int nc = p.nc;
    double *cols = tile + p.col0 * p.pitch;
    const int pad = p.pitch - nc;
    for (int e = threadIdx.x; e < nc * pad; e += blockDim.x) cols[(int64_t)(e / pad) * p.pitch + nc + e % pad] = 0.0;
    for (int e = threadIdx.x; e < p.col0 * p.pitch; e += blockDim.x) tile[e] = 0.0;
    if (p.dx) { // <dx_ci, dx_cj>: a warp takes 8 columns, its lanes the rows
        const double *dx = p.dx + b * p.d * nc;
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, warps = blockDim.x >> 5;
        for (int cj = w * 8; cj < nc; cj += warps * 8) {
            for (int ci = lane; ci < nc; ci += 32) {
                double acc[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[j] = 0.0;
#pragma unroll 2
                for (int64_t k = 0; k < p.d; ++k) {
                    const double *row = dx + k * nc;
                    const double a = row[ci];
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[j] = fma(a, row[cj + j < nc ? cj + j : cj], acc[j]);
                }
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (cj + j < nc) cols[(int64_t)(cj + j) * p.pitch + ci] = acc[j];
            }
        }
    } else { // the caller's, threads along the axis that is contiguous
        const bool rows = p.is1 <= p.is2;
        for (int64_t e = threadIdx.x; e < (int64_t)nc * nc; e += blockDim.x) {
            const int64_t hi = e / nc, lo = e - hi * nc;
            const int64_t ci = rows ? lo : hi, cj = rows ? hi : lo;
            const int64_t at = b * p.is0 + ci * p.is1 + cj * p.is2;
            cols[cj * p.pitch + ci] = p.in64 ? reinterpret_cast<const double *>(p.inc)[at]
                                             : (double)reinterpret_cast<const float *>(p.inc)[at];
        }
    }
}

// K[n][n] of the path on increments tile * f, in every thread of the solving
// warps; s_val is the CTA's word for it.
//
// With one warp a sub-partition, time goes with the instruction stream and its
// dependences, not with throughput: with bound checks and indexes computed each
// step a step of 2 x 2 cells took 440 cycles.  So the loop has no branches on a
// lane's place.  Before its first column a lane runs with increments 0 on ones,
// which gives 1 exactly; after its last one it runs on, and the run ends with
// the step that finishes row n.  A step's coefficients are formed during the
// step before, from increments loaded PF steps earlier.
// P: NormParams, or another kernel's parameters with the same geometry (nc: rows
// of the pair).  CHAIN: one dependent operation a cell down a column instead of
// two; without it the cells are those of stencil_cell, bit for bit.
template <int R, int O, bool SMEM, bool BSMEM, bool CHAIN, class P>
__device__ __forceinline__ double norm_solve(const P &p, const double *tile, double *bnd, double f,
                                             double *s_val)
{
    using NS = NormShape<R, O>;
    constexpr int C = NS::C, RC = NS::RC, CC = NS::CC, PF = NS::ahead(SMEM);
    constexpr int LEAD = (PF + 1 + kNormChunk - 1) / kNormChunk * kNormChunk; // steps that fill the pipeline
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int nsteps = p.nsteps, row = nsteps * C;
    const int last = (p.nc << p.order) - 1 - (p.nbands - 1) * 32 * R; // last row within its band
    const int lstar = last / R, rstar = last % R;
    const int zeros = (p.nc + RC - 1) / RC * RC; // rows from here on are zeros
    double res = 1.0;
    for (int b0 = 0; b0 < p.nbands; b0 += p.nw) {
        const int b = b0 + w;
        const bool mine = b < p.nbands;
        const bool ends = b0 + p.nw >= p.nbands; // the last group ends with row n, others with lane 31
        const int wl = ends ? p.nbands - 1 - b0 : p.nw - 1;
        int total = LEAD + wl * kNormLag + nsteps + (ends ? lstar : 31);
        const int pad = (kNormChunk - total % kNormChunk) % kNormChunk;
        total += pad;
        const int begin = LEAD + pad + w * kNormLag; // lane 0's first step of the run
        const int ci0 = ((b * 32 + lane) * R) >> p.order;
        NormMem<SMEM> rows(tile + (ci0 < zeros ? ci0 : zeros)); // the lane's rows of the next column to load
        // the row above (row 0 of bnd: ones, for the first band) and the row below
        NormMem<BSMEM> above(b == 0 ? bnd : bnd + C + (w == 0 ? p.nw - 1 : w - 1) * row), below(bnd + C + w * row);
        const bool writes = lane == 31 && b + 1 < p.nbands;
        int q = -begin - lane;
        double left[R], bot[C], tn[C], corner = 1.0;
        double A[CC][RC], B[CC][RC], cn[PF][CC][RC];
#pragma unroll
        for (int r = 0; r < R; ++r) left[r] = 1.0;
#pragma unroll
        for (int c = 0; c < C; ++c) {
            bot[c] = 1.0;
            tn[c] = 1.0;
        }
#pragma unroll
        for (int cc = 0; cc < CC; ++cc)
#pragma unroll
            for (int rc = 0; rc < RC; ++rc) {
                A[cc][rc] = 1.0;
                B[cc][rc] = 1.0;
#pragma unroll
                for (int i = 0; i < PF; ++i) cn[i][cc][rc] = 0.0;
            }
        for (int s = 0; s < total; s += kNormChunk) {
            if (mine && s >= begin - LEAD - pad && s < begin + nsteps + 31) { // warp-uniform
#pragma unroll
                for (int j = 0; j < kNormChunk; ++j) {
                    double top[C];
#pragma unroll
                    for (int c = 0; c < C; ++c) top[c] = __shfl_up_sync(kFullMask, bot[c], 1);
#pragma unroll
                    for (int c = 0; c < C; ++c) top[c] = lane == 0 ? tn[c] : top[c];
#pragma unroll
                    for (int c = 0; c < C; ++c) {
                        const int cc = NS::cc_of(c);
                        double up = top[c], dg = c == 0 ? corner : top[c > 0 ? c - 1 : 0];
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            const double l = left[r], a = A[cc][NS::rc_of(r)], bb = B[cc][NS::rc_of(r)];
                            up = CHAIN ? stencil_chain(dg, up, l, a, bb) : stencil_cell(dg, up, l, a, bb);
                            dg = l;
                            left[r] = up;
                        }
                        bot[c] = up;
                    }
                    corner = top[C - 1];
                    const bool was = (unsigned)q < (unsigned)nsteps;
#pragma unroll
                    for (int c = 0; c < C; c += 2) below.put2(c, bot[c], bot[c + 1], writes && was);
                    below.move(was ? C : 0);
                    ++q;
                    // lane 0's next row above: ones until its first step and after its last one
                    const bool in = (unsigned)q < (unsigned)nsteps;
#pragma unroll
                    for (int c = 0; c < C; c += 2) {
                        const double2 v = above.get2(c);
                        tn[c] = in ? v.x : 1.0;
                        tn[c + 1] = in ? v.y : 1.0;
                    }
                    above.move(in && b > 0 ? C : 0);
                    // An infinite increment times 0 is NaN: a root-find takes the NaN of its path for an overflow either
                    // way, and a selection a coefficient cost it 3%; a pair's own value may be infinite.
                    const double fq = in ? f : 0.0;
#pragma unroll
                    for (int cc = 0; cc < CC; ++cc)
#pragma unroll
                        for (int rc = 0; rc < RC; ++rc) {
                            const double v = cn[j % PF][cc][rc];
                            stencil_coefs(CHAIN ? v * fq : in ? v * f : 0.0, A[cc][rc], B[cc][rc]);
                        }
                    // increments of step q + PF; `rows` stays inside the columns
                    const int qn = q + PF;
                    NormMem<SMEM> src = rows;
                    if constexpr (!NS::WHOLE)
                        src.move(norm_col_offset(qn, nsteps, C, p.order, p.pitch));
#pragma unroll
                    for (int cc = 0; cc < CC; ++cc) {
                        if constexpr (RC == 1) {
                            cn[j % PF][cc][0] = src.get(0);
                        } else {
#pragma unroll
                            for (int rc = 0; rc < RC; rc += 2) {
                                const double2 v = src.get2(rc);
                                cn[j % PF][cc][rc] = v.x;
                                cn[j % PF][cc][rc + 1] = v.y;
                            }
                        }
                        if (cc + 1 < CC) src.move(p.pitch);
                    }
                    if constexpr (NS::WHOLE) rows.move((unsigned)qn < (unsigned)(nsteps - 1) ? CC * p.pitch : 0);
                }
            } else {
                q += kNormChunk;
            }
            norm_barrier(p.nw);
        }
        if (ends) {
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (r == rstar) res = left[r];
        }
    }
    res = __shfl_sync(kFullMask, res, lstar);
    if (p.nw == 1) return res;
    if (w == (p.nbands - 1) % p.nw && lane == 0) *s_val = res;
    norm_barrier(p.nw);
    res = *s_val;
    norm_barrier(p.nw); // s_val and the rows are free for the next solve
    return res;
}

// blockDim: the solving warps, and more to help with the tile where there are
// fewer than four.
template <int R, int O, bool SMEM, bool BSMEM>
__global__ void __launch_bounds__(NormShape<R, O>::MAXW * 32, 1) norm_kernel(NormParams p)
{
    using NS = NormShape<R, O>;
    extern __shared__ __align__(16) double norm_smem[];
    __shared__ double s_val;
    double *tile = SMEM ? norm_smem : p.tiles + blockIdx.x * p.tile;
    const int rows = norm_bnd_values(p.nbands, p.nw, p.nsteps, NS::C);
    double *bnd = BSMEM ? norm_smem + (SMEM ? p.tile : 0) : p.bnd + (int64_t)blockIdx.x * rows;
    if (threadIdx.x < NS::C) bnd[threadIdx.x] = 1.0;
    for (int64_t b = blockIdx.x; b < p.n; b += gridDim.x) {
        norm_build_tile(p, b, tile);
        __syncthreads();
        if ((threadIdx.x >> 5) < p.nw) {
            auto solve = [&](double scale) -> double {
                return norm_solve<R, O, SMEM, BSMEM, true>(p, tile, bnd, p.fscale * scale, &s_val);
            };
            double out = 0.0;
            int it = 0;
            normalize_path(p, b, threadIdx.x == 0, solve, out, it);
            if (threadIdx.x == 0) {
                if (p.lam) {
                    if (p.in64)
                        reinterpret_cast<double *>(p.lam)[b] = out;
                    else
                        reinterpret_cast<float *>(p.lam)[b] = (float)out;
                }
                if (p.iters) p.iters[b] = it;
            }
        }
        __syncthreads(); // the tile is free for the next path
    }
}

} // namespace sigk
