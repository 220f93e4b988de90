// Backward pass: gradients of sum_pairs w * k(x, y) with respect to the path
// points, for the linear static kernel with float64 cells.  The reference has
// no backward pass (its Numba kernels end autograd); this is the adjoint of
// the same scheme (sigpde/cuda_device_functions.py:3-5).
//
// With c the scaled coarse increment of a cell, A(c) = 1 + c/2 + c^2/12 and
// B(c) = 1 - c^2/12, the forward scheme is
//   K(p,q) = (K(p,q-1) + K(p-1,q)) A - K(p-1,q-1) B.
// Its adjoint Lambda = w dk/dK(p,q) satisfies, in reverse order,
//   Lambda(p,q) = P(p,q+1) + P(p+1,q) - Q(p+1,q+1),   Lambda(n,m) = w,
// where each node carries P = A Lambda and Q = B Lambda with the coefficients
// of the cell that produced it (absent nodes carry 0), and
//   dk/dc of a coarse cell = sum over its fine cells of Lambda(p,q) D(p,q),
//   D(p,q) = (K(p,q-1) + K(p-1,q)) A'(c) - K(p-1,q-1) B'(c),
//   A'(c) = 1/2 + c/6,  B'(c) = -c/6.
//
// Kernels
//   grad_fwd_kernel  the forward wavefront over a run of pairs a warp, writing
//                    what enters every lane step: the values above the
//                    lane's block, left of it and above-left of it;
//   grad_bwd_kernel  the same lane steps in reverse time: each lane recomputes
//                    its block's D from that record alone (no other lane is
//                    asked), then runs the adjoint over the block, summing
//                    Lambda D per coarse cell; each coarse cell's rows belong
//                    to one lane (R >= 2^order), so the sum is written once,
//                    over the cell's increment in the increment matrix (which
//                    then holds dk/dc);
//   grad_gx_kernel / grad_gy_kernel   contractions of dk/dc with the scaled
//                    differences of the other side: the gradients with
//                    respect to the coarse differences;
//   grad_points_kernel   their partial sums, and the differences of those: gradients at the points;
//   grad_stage_kernel    the scaled differences in every layout that these read.
#pragma once

#include "dgemm_inc.cuh"

namespace sigk {

struct GradParams {
    int op;               // kOpPairwise / kOpGram
    double *mat;          // increments in, dk/dc out; Gram: [n * ld + m], pairwise: per-pair blocks
    int64_t ld;           // Gram: npaths_x(chunk) * rows_x; pairwise: rows_x
    int64_t rows_x;
    int64_t ncx, ncy;
    int order;
    int64_t nitems;       // pairs in this chunk
    int64_t per_warp;     // pairs a warp (a contiguous run)
    int nb, nsteps, period; // bands a pair, lane steps a band, steps from one band's start to the next
    int64_t ny;           // Gram: y paths
    const void *w;        // weights (grad_out): pairwise (n,), Gram (n_x, n_y) row-major; input dtype
    int in64;
    int64_t x0;           // first x path of the chunk
    double *rec;          // per warp grad_warp_steps(...) records of what enters its lane steps
    double *bnd;          // per warp bnd_stride doubles: rows handed from band to band
    int64_t bnd_stride;
    int bnd_smem;         // forward: those rows are in dynamic shared memory instead
};

// Lane-step shape.  A lane owns R rows and takes C columns a step: the cells of
// an R x C block are independent along anti-diagonals, and a step's loads,
// shuffles, control and record are paid once for all of them (one column a step
// with the same R spent 33 instructions a cell, 10 of them float64; the adjoint
// then ran at 35% of the float64 pipe).  A block's D stays in registers: 32
// cells at three CTAs an SM (W = 1), or 64 at two (W = 2, long runs: 128 x 128
// pairs, L = 128, order 2 run 4.12 + 2.25 ms backward + forward against
// 4.64 + 3.13, with 4 columns; short runs pay the wider pipeline fill).  Orders
// 3 and 4 may split a coarse column over several steps; orders 0 and 1 take
// several whole coarse columns a step.
template <int R, int O, int W>
struct GradShape {
    static constexpr int C = (O == 0 || O == 4) ? 2 : 4 * W;
    static constexpr int RC = R >> O;                        // coarse rows a lane
    static constexpr int CC = (C >> O) > 0 ? (C >> O) : 1;   // coarse columns a step
    static constexpr bool WHOLE = (C >> O) > 0;              // steps hold whole coarse columns
    static constexpr int NV2 = (R + C) / 2;                  // 16-byte parts of a lane step's record
    static constexpr int REC = NV2 * 64 + 32;                // doubles of a warp step's record
    static constexpr int INC = CC * RC * 32;                 // doubles of a warp step's increments
    static constexpr int CTAS = W == 1 ? 3 : 2;              // resident CTAs an SM
    static_assert(R >= (1 << O) && R % 2 == 0 && C % 2 == 0, "a lane's rows hold whole coarse rows");
    __host__ __device__ static constexpr int cc_of(int c) { return CC == 1 ? 0 : c >> O; }
};

// Warp schedule, shared by both kernels (the backward kernel runs it in
// reverse).  A warp walks a run of pairs, each in nb bands of 32 R rows; lane
// l does step q of the run's v-th band at warp step s = v * period + q + l, so
// the lane pipeline does not drain between bands and pairs.  A band needs the
// row that lane 31 of the band above wrote 31 steps after lane 0 took the same
// columns: with several bands the period is at least kGradMinPeriod, which
// leaves room to load that row one step ahead.
constexpr int kGradMinPeriod = 34;
constexpr int kGradFwdRing = 4; // steps of increments in shared memory: one in use, three in flight
constexpr int kGradRing = 3;    // backward: one step of records and increments in use, two in flight

__host__ __device__ __forceinline__ int64_t grad_warp_steps(int64_t pairs, int nb, int period)
{
    return pairs * nb * period + 31;
}

template <int R, int O, int W>
constexpr size_t grad_bwd_smem()
{
    using GS = GradShape<R, O, W>;
    return (size_t)kWarpsPerBlock * kGradRing * (GS::REC + GS::INC) * sizeof(double);
}

// A lane's place in the warp's run: step q of the period (idle from nsteps on),
// band b and pair (yj, and the first of its own coarse rows in the pair's
// increment block).
struct GradPos {
    int q, b;
    int64_t yj;
    double *rows; // increment (ci0, 0) of the band's coarse rows ci0 of this lane
    int ci0;
};

template <int R, int O>
__device__ __forceinline__ GradPos grad_pos(const GradParams &p, int64_t it, int b, int q, int lane)
{
    GradPos w;
    const int64_t xi = p.op == kOpPairwise ? it : it / p.ny;
    w.yj = p.op == kOpPairwise ? 0 : it - xi * p.ny;
    w.q = q;
    w.b = b;
    w.ci0 = ((b * 32 + lane) * R) >> O;
    w.rows = (p.op == kOpPairwise ? p.mat + it * p.ncy * p.rows_x : p.mat + w.yj * p.ncy * p.ld + xi * p.rows_x) + w.ci0;
    return w;
}

// the band after (q is the caller's)
template <int R, int O>
__device__ __forceinline__ void grad_next_band(const GradParams &p, GradPos &w, int lane)
{
    w.rows += (32 * R) >> O;
    w.ci0 += (32 * R) >> O;
    if (++w.b < p.nb) return;
    w.b = 0;
    w.rows -= w.ci0; // back to the pair's first rows
    w.ci0 = (lane * R) >> O;
    w.rows += w.ci0;
    if (p.op == kOpPairwise) {
        w.rows += p.ncy * p.rows_x;
    } else if (++w.yj < p.ny) {
        w.rows += p.ncy * p.ld;
    } else {
        w.yj = 0;
        w.rows += p.rows_x - (p.ny - 1) * p.ncy * p.ld;
    }
}

// the band before
template <int R, int O>
__device__ __forceinline__ void grad_prev_band(const GradParams &p, GradPos &w, int lane)
{
    w.rows -= (32 * R) >> O;
    w.ci0 -= (32 * R) >> O;
    if (--w.b >= 0) return;
    w.b = p.nb - 1;
    w.rows -= w.ci0;
    w.ci0 = ((w.b * 32 + lane) * R) >> O;
    w.rows += w.ci0;
    if (p.op == kOpPairwise) {
        w.rows -= p.ncy * p.rows_x;
    } else if (--w.yj >= 0) {
        w.rows -= p.ncy * p.ld;
    } else {
        w.yj = p.ny - 1;
        w.rows += (p.ny - 1) * p.ncy * p.ld - p.rows_x;
    }
}

__device__ __forceinline__ void grad_cp_async16(void *dst, const void *src)
{
    const unsigned a = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(src) : "memory");
}

// n bytes copied, the rest of the 16 (8) filled with 0
__device__ __forceinline__ void grad_cp_async16z(void *dst, const void *src, int n)
{
    const unsigned a = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(a), "l"(src), "r"(n) : "memory");
}

__device__ __forceinline__ void grad_cp_async8z(void *dst, const void *src, int n)
{
    const unsigned a = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(a), "l"(src), "r"(n) : "memory");
}

// The increments of a lane step (CC coarse columns of RC rows) come through a
// shared-memory ring several steps ahead: one step ahead in registers left the
// forward pass waiting on HBM (37% of its issue bound).  Cells beyond the
// pair's rows and columns, and steps outside the run (`run` false), are filled
// with 0; a path's rows are padded to a multiple of 4 with zeros, so a 16-byte
// copy that starts inside a path stays inside its padding.
template <int R, int O, int W>
__device__ __forceinline__ void grad_fetch_incs(const GradParams &p, const GradPos &w, bool run, int64_t row_ld,
                                                double *slot, int lane)
{
    using GS = GradShape<R, O, W>;
    run = run && w.q < p.nsteps;
    const int cj0 = (w.q * GS::C) >> O;
#pragma unroll
    for (int cc = 0; cc < GS::CC; ++cc) {
        const bool in = run && cj0 + cc < (int)p.ncy;
        const double *col = w.rows + (int64_t)(cj0 + cc) * row_ld;
        if constexpr (GS::RC == 1) {
            const bool ok = in && w.ci0 < (int)p.ncx;
            grad_cp_async8z(slot + cc * 32 + lane, ok ? col : p.mat, ok ? 8 : 0);
        } else {
#pragma unroll
            for (int h = 0; h < GS::RC / 2; ++h) {
                const bool ok = in && w.ci0 + 2 * h < (int)p.ncx;
                grad_cp_async16z(slot + 2 * ((cc * (GS::RC / 2) + h) * 32 + lane), ok ? col + 2 * h : p.mat, ok ? 16 : 0);
            }
        }
    }
}

template <int R, int O, int W>
__device__ __forceinline__ void grad_read_incs(const double *slot, int lane,
                                               double (&c)[GradShape<R, O, W>::CC][GradShape<R, O, W>::RC])
{
    using GS = GradShape<R, O, W>;
#pragma unroll
    for (int cc = 0; cc < GS::CC; ++cc) {
        if constexpr (GS::RC == 1) {
            c[cc][0] = slot[cc * 32 + lane];
        } else {
#pragma unroll
            for (int h = 0; h < GS::RC / 2; ++h) {
                const double2 v = *reinterpret_cast<const double2 *>(slot + 2 * ((cc * (GS::RC / 2) + h) * 32 + lane));
                c[cc][2 * h] = v.x;
                c[cc][2 * h + 1] = v.y;
            }
        }
    }
}

// grad_fwd_kernel is bound by its record: (R + C + 1) / (R C) doubles a cell,
// written once, against 3 float64 operations (128 x 128 pairs, L = 128, order 2:
// 9.1 GB in 2.26 ms; the kernel before it, one column a step, took 3.48 ms).
template <int R, int O, int W>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, (GradShape<R, O, W>::CTAS)) grad_fwd_kernel(GradParams p)
{
    using GS = GradShape<R, O, W>;
    constexpr int C = GS::C, RC = GS::RC, CC = GS::CC;
    extern __shared__ __align__(16) unsigned char grad_smem[]; // the warps' boundary rows, if they fit
    __shared__ __align__(16) double incs[kWarpsPerBlock][kGradFwdRing][GS::INC];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int64_t gwarp = (int64_t)blockIdx.x * kWarpsPerBlock + wib;
    const int64_t first = gwarp * p.per_warp;
    if (first >= p.nitems) return; // warp-uniform
    const int cnt = (int)(p.nitems - first < p.per_warp ? p.nitems - first : p.per_warp);
    const int nsteps = p.nsteps, period = p.period;
    const int64_t row_ld = p.op == kOpPairwise ? p.rows_x : p.ld;
    const int run = cnt * p.nb * period, steps = run + 31;
    double *rec = p.rec + gwarp * grad_warp_steps(p.per_warp, p.nb, period) * GS::REC;
    // K of the row above the next band, columns 1..nsteps * C
    double *bnd = p.bnd_smem ? reinterpret_cast<double *>(grad_smem) + wib * nsteps * C : p.bnd + gwarp * p.bnd_stride;
    double(*ring)[GS::INC] = incs[wib];

    GradPos w = grad_pos<R, O>(p, first, 0, 0, lane), f = w; // f: the step whose increments are fetched
    auto fetch = [&](int s) { // of warp step s; called for s = 0, 1, ...
        if (s >= lane) {
            grad_fetch_incs<R, O, W>(p, f, s - lane < run, row_ld, ring[s & (kGradFwdRing - 1)], lane);
            if (++f.q == period) {
                f.q = 0;
                grad_next_band<R, O>(p, f, lane);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0);
    fetch(1);
    fetch(2);
    double tn[C]; // lane 0: the row above its next step
    double left[R], bot[C], corner = 1.0;
#pragma unroll
    for (int r = 0; r < R; ++r) left[r] = 1.0;
#pragma unroll
    for (int c = 0; c < C; ++c) {
        bot[c] = 1.0;
        tn[c] = 1.0;
    }
    for (int s = 0; s < steps; ++s) {
        fetch(s + 3);
        asm volatile("cp.async.wait_group 3;" ::: "memory"); // step s has arrived
        double top[C];
#pragma unroll
        for (int c = 0; c < C; ++c) top[c] = __shfl_up_sync(kFullMask, bot[c], 1);
        if (lane == 0) {
#pragma unroll
            for (int c = 0; c < C; ++c) top[c] = tn[c];
        }
        if ((unsigned)(s - lane) < (unsigned)run) {
            if (w.q < nsteps) {
                double A[CC][RC], B[CC][RC];
                grad_read_incs<R, O, W>(ring[s & (kGradFwdRing - 1)], lane, A);
#pragma unroll
                for (int cc = 0; cc < CC; ++cc)
#pragma unroll
                    for (int rc = 0; rc < RC; ++rc) stencil_coefs(A[cc][rc], A[cc][rc], B[cc][rc]);
                double *rs = rec + (int64_t)s * GS::REC;
                double2 *rs2 = reinterpret_cast<double2 *>(rs) + lane;
#pragma unroll
                for (int c = 0; c < C / 2; ++c) __stcs(rs2 + c * 32, make_double2(top[2 * c], top[2 * c + 1]));
#pragma unroll
                for (int r = 0; r < R / 2; ++r) __stcs(rs2 + (C / 2 + r) * 32, make_double2(left[2 * r], left[2 * r + 1]));
                __stcs(rs + GS::NV2 * 64 + lane, corner);
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    const int cc = GS::cc_of(c);
                    double up = top[c], dg = c == 0 ? corner : top[c - 1];
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const double l = left[r], a = A[cc][r >> O];
                        up = fma(up, a, fma(l, a, -(dg * B[cc][r >> O])));
                        dg = l;
                        left[r] = up;
                    }
                    bot[c] = up;
                }
                corner = top[C - 1];
                if (lane == 31 && w.b + 1 < p.nb) {
#pragma unroll
                    for (int c = 0; c < C; ++c) bnd[w.q * C + c] = bot[c];
                }
            }
            if (++w.q == period) { // the next band starts
                w.q = 0;
                grad_next_band<R, O>(p, w, lane);
#pragma unroll
                for (int r = 0; r < R; ++r) left[r] = 1.0;
                corner = 1.0;
            }
            if (lane == 0 && w.q < nsteps) {
#pragma unroll
                for (int c = 0; c < C; ++c) tn[c] = w.b > 0 ? bnd[w.q * C + c] : 1.0;
            }
        }
        __syncwarp(); // orders lane 31's boundary stores before lane 0's loads
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// grad_bwd_kernel: per cell 5 float64 operations for D (K of the block and
// dK/dc in one pass), 3 for Lambda and 1 for the sum.  The record and the
// increments come through shared-memory rings of cp.async copies, two steps
// ahead.  Lambda of a cell is
//   A(right) Lambda(right) + A(below) Lambda(below) - B(diagonal) Lambda(diagonal),
// three operations with the coefficients of the three cells' coarse cells:
// those of the column to the right are kept from the previous step (AR, BR),
// those of the row below come from lane l + 1 with its Lambda.  An SM
// sub-partition issues a float64 instruction in two slots and any other in one,
// so the bound is 18 slots a cell plus the step's rest; 128 x 128 pairs,
// L = 128, order 2: 4.20 ms, 2.05 of them float64 (one column a step: 9.48 ms).
template <int R, int O, int W>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, (GradShape<R, O, W>::CTAS)) grad_bwd_kernel(GradParams p)
{
    using GS = GradShape<R, O, W>;
    constexpr int C = GS::C, RC = GS::RC, CC = GS::CC, NV2 = GS::NV2;
    extern __shared__ __align__(16) unsigned char grad_smem[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int64_t gwarp = (int64_t)blockIdx.x * kWarpsPerBlock + wib;
    const int64_t first = gwarp * p.per_warp;
    if (first >= p.nitems) return; // warp-uniform
    const int cnt = (int)(p.nitems - first < p.per_warp ? p.nitems - first : p.per_warp);
    const int ncx = (int)p.ncx, ncy = (int)p.ncy, nsteps = p.nsteps, period = p.period;
    const int n = ncx << O;
    const int64_t row_ld = p.op == kOpPairwise ? p.rows_x : p.ld;
    const int run = cnt * p.nb * period, steps = run + 31;
    const double *rec = p.rec + gwarp * grad_warp_steps(p.per_warp, p.nb, period) * GS::REC;
    double *ring = reinterpret_cast<double *>(grad_smem) + wib * kGradRing * (GS::REC + GS::INC);
    // the first row of the band below: Lambda of its columns, then A and B of its coarse columns
    double *bL = p.bnd + gwarp * p.bnd_stride, *bA = bL + nsteps * C, *bB = bA + nsteps * CC;

    GradPos w = grad_pos<R, O>(p, first + cnt - 1, p.nb - 1, period - 1, lane), f = w;
    int64_t wi = (p.op == kOpPairwise ? p.x0 : p.x0 * p.ny) + first + cnt - 1; // the pair's weight
    auto fetch = [&](int s, int slot) { // of warp step s; called for s = steps - 1, steps - 2, ...
        double *dst = ring + slot * (GS::REC + GS::INC);
        if (s >= 0) {
            const double *src = rec + (int64_t)s * GS::REC;
#pragma unroll
            for (int i = 0; i < NV2; ++i) grad_cp_async16(dst + 2 * (i * 32 + lane), src + 2 * (i * 32 + lane));
            grad_cp_async8z(dst + NV2 * 64 + lane, src + NV2 * 64 + lane, 8);
        }
        if (s - lane < run) {
            grad_fetch_incs<R, O, W>(p, f, s >= lane, row_ld, dst + GS::REC, lane);
            if (--f.q < 0) {
                f.q = period - 1;
                grad_prev_band<R, O>(p, f, lane);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(steps - 1, 0);
    fetch(steps - 2, 1);
    int slot = 0;

    double Lr[R];                        // Lambda of the lane's rows at the column right of the block
    double AR[RC], BR[RC], bBR;          // A, B of that column (bBR: B of the row below)
    double g[CC][RC];
    double topL[C], tA[CC], tB[CC];     // Lambda and coefficients of the lane's first row, for lane l - 1
    double below0;                       // Lambda below-right of the block
    auto start_band = [&]() { // nothing lies to the right of the band's last column
        const int rseed = w.b == p.nb - 1 ? n - 1 - (w.b * 32 + lane) * R : -1;
        double wt = 0.0;
        if (rseed >= 0 && rseed < R) // Lambda(n, m) = the pair's weight, as row n's right neighbour
            wt = p.in64 ? reinterpret_cast<const double *>(p.w)[wi] : (double)reinterpret_cast<const float *>(p.w)[wi];
#pragma unroll
        for (int r = 0; r < R; ++r) Lr[r] = r == rseed ? wt : 0.0;
#pragma unroll
        for (int rc = 0; rc < RC; ++rc) {
            AR[rc] = 1.0;
            BR[rc] = 0.0;
        }
        bBR = 0.0;
        below0 = 0.0;
    };
    start_band();
#pragma unroll
    for (int c = 0; c < C; ++c) topL[c] = 0.0;
#pragma unroll
    for (int cc = 0; cc < CC; ++cc) {
        tA[cc] = 1.0;
        tB[cc] = 1.0;
#pragma unroll
        for (int rc = 0; rc < RC; ++rc) g[cc][rc] = 0.0;
    }

    for (int s = steps - 1; s >= 0; --s) {
        fetch(s - 2, slot == 0 ? kGradRing - 1 : slot - 1); // the slot of step s + 1
        asm volatile("cp.async.wait_group 2;" ::: "memory"); // step s has arrived
        double bl[C], bAc[CC], bBc[CC]; // the row below: Lambda and coefficients
#pragma unroll
        for (int c = 0; c < C; ++c) bl[c] = __shfl_down_sync(kFullMask, topL[c], 1);
#pragma unroll
        for (int cc = 0; cc < CC; ++cc) {
            bAc[cc] = __shfl_down_sync(kFullMask, tA[cc], 1);
            bBc[cc] = __shfl_down_sync(kFullMask, tB[cc], 1);
        }
        if ((unsigned)(s - lane) < (unsigned)run) {
            if (w.q < nsteps) {
                if (lane == 31) {
                    const bool has = w.b + 1 < p.nb;
#pragma unroll
                    for (int c = 0; c < C; ++c) bl[c] = has ? bL[w.q * C + c] : 0.0;
#pragma unroll
                    for (int cc = 0; cc < CC; ++cc) {
                        bAc[cc] = has ? bA[w.q * CC + cc] : 1.0;
                        bBc[cc] = has ? bB[w.q * CC + cc] : 1.0;
                    }
                }
                const double *rs = ring + slot * (GS::REC + GS::INC);
                double A[CC][RC], B[CC][RC], Ad[CC][RC], Bd[CC][RC];
                grad_read_incs<R, O, W>(rs + GS::REC, lane, A);
#pragma unroll
                for (int cc = 0; cc < CC; ++cc)
#pragma unroll
                    for (int rc = 0; rc < RC; ++rc) {
                        const double c = A[cc][rc];
                        stencil_coefs(c, A[cc][rc], B[cc][rc]);
                        Ad[cc][rc] = fma(c, 1.0 / 6.0, 0.5);
                        Bd[cc][rc] = c * (1.0 / 6.0); // -B'
                    }
                double D[R][C];
                { // D of the block from the record
                    double left[R], top[C];
                    const double2 *rs2 = reinterpret_cast<const double2 *>(rs) + lane;
#pragma unroll
                    for (int c = 0; c < C / 2; ++c) {
                        const double2 v = rs2[c * 32];
                        top[2 * c] = v.x;
                        top[2 * c + 1] = v.y;
                    }
#pragma unroll
                    for (int r = 0; r < R / 2; ++r) {
                        const double2 v = rs2[(C / 2 + r) * 32];
                        left[2 * r] = v.x;
                        left[2 * r + 1] = v.y;
                    }
                    const double corner = rs[NV2 * 64 + lane];
#pragma unroll
                    for (int c = 0; c < C; ++c) {
                        const int cc = GS::cc_of(c);
                        double up = top[c], dg = c == 0 ? corner : top[c > 0 ? c - 1 : 0];
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            const int rc = r >> O;
                            const double l = left[r], sum = l + up;
                            D[r][c] = fma(sum, Ad[cc][rc], dg * Bd[cc][rc]);
                            up = fma(sum, A[cc][rc], -(dg * B[cc][rc]));
                            dg = l;
                            left[r] = up;
                        }
                    }
                }
#pragma unroll
                for (int c = C - 1; c >= 0; --c) {
                    const bool edge_r = c == C - 1;
                    const int cc = GS::cc_of(c), cr = edge_r ? 0 : GS::cc_of(c + 1);
                    double dn = bl[c], dgl = edge_r ? below0 : bl[edge_r ? 0 : c + 1];
#pragma unroll
                    for (int r = R - 1; r >= 0; --r) {
                        const bool edge_d = r == R - 1;
                        const int rc = r >> O, rb = edge_d ? 0 : (r + 1) >> O; // rb: coarse row below
                        const double ad = edge_d ? bAc[cc] : A[cc][rb];
                        const double ar = edge_r ? AR[rc] : A[cr][rc];
                        const double bg = edge_r ? (edge_d ? bBR : BR[rb]) : (edge_d ? bBc[cr] : B[cr][rb]);
                        const double lr = Lr[r];
                        const double lam = fma(ad, dn, fma(ar, lr, -(bg * dgl)));
                        // the coarse cell's first fine cell in this order starts its sum
                        const bool starts = GS::WHOLE && (edge_d || rc != rb) && (edge_r || cc != cr);
                        g[cc][rc] = starts ? lam * D[r][c] : fma(lam, D[r][c], g[cc][rc]);
                        dgl = lr;
                        dn = lam;
                        Lr[r] = lam;
                    }
                    topL[c] = dn;
                }
                below0 = bl[0];
                bBR = bBc[0];
#pragma unroll
                for (int rc = 0; rc < RC; ++rc) {
                    AR[rc] = A[0][rc];
                    BR[rc] = B[0][rc];
                }
#pragma unroll
                for (int cc = 0; cc < CC; ++cc) {
                    tA[cc] = A[cc][0];
                    tB[cc] = B[cc][0];
                }
                if (lane == 0 && w.b > 0) {
#pragma unroll
                    for (int c = 0; c < C; ++c) bL[w.q * C + c] = topL[c];
#pragma unroll
                    for (int cc = 0; cc < CC; ++cc) {
                        bA[w.q * CC + cc] = tA[cc];
                        bB[w.q * CC + cc] = tB[cc];
                    }
                }
                if (GS::WHOLE || ((w.q * C) & ((1 << O) - 1)) == 0) { // dk/dc of the coarse columns is complete
                    const int cj0 = (w.q * C) >> O;
#pragma unroll
                    for (int cc = 0; cc < CC; ++cc) {
                        double *col = w.rows + (int64_t)(cj0 + cc) * row_ld;
                        if (CC == 1 || cj0 + cc < ncy) {
                            if constexpr (RC == 1) {
                                if (w.ci0 < ncx) col[0] = g[cc][0];
                            } else {
#pragma unroll
                                for (int h = 0; h < RC / 2; ++h) {
                                    if (w.ci0 + 2 * h + 1 < ncx)
                                        *reinterpret_cast<double2 *>(col + 2 * h) = make_double2(g[cc][2 * h], g[cc][2 * h + 1]);
                                    else if (w.ci0 + 2 * h < ncx)
                                        col[2 * h] = g[cc][2 * h];
                                }
                            }
                        }
                        if constexpr (!GS::WHOLE) {
#pragma unroll
                            for (int rc = 0; rc < RC; ++rc) g[cc][rc] = 0.0;
                        }
                    }
                }
            }
            if (--w.q < 0) {
                w.q = period - 1;
                if (w.b == 0) --wi;
                grad_prev_band<R, O>(p, w, lane);
                if (s > lane) start_band();
            }
        }
        slot = slot == kGradRing - 1 ? 0 : slot + 1;
        __syncwarp(); // orders lane 0's boundary stores before lane 31's loads
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// Increments of pairwise pairs (x path = y path = x0 + item) in per-pair
// blocks [item][cj][ci] (ci < rows_x; rows ci >= ncx are 0), summed as
// fma(dx_k, dy_k, acc) for k = 0 .. d-1 from zero like the other producers.
template <int V = 0> // instantiated once, in kernels_grad.cu
__global__ void grad_pair_inc_kernel(const double *dx, const double *dy, int64_t nitems, int64_t x0, int64_t ncx,
                                     int64_t ncy, int64_t rows_x, int64_t d, double *out)
{
    const int64_t total = nitems * ncy * rows_x;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t item = e / (ncy * rows_x), r = e - item * ncy * rows_x;
        const int64_t cj = r / rows_x, ci = r - cj * rows_x;
        double acc = 0.0;
        if (ci < ncx) {
            const double *a = dx + (x0 + item) * d * ncx + ci;
            const double *b = dy + (x0 + item) * d * ncy + cj;
            for (int64_t k = 0; k < d; ++k) acc = fma(a[k * ncx], b[k * ncy], acc);
        }
        out[e] = acc;
    }
}

// Caller's increments (npairs, ncx, ncy) with element strides, times the
// pair's scales, into per-pair blocks [item][cj][ci] (rows ci >= ncx are 0);
// with `back`, the reverse: out = block * scales written with the strides.
template <int V = 0> // instantiated once, in kernels_grad.cu
__global__ void grad_inc_blocks_kernel(const void *inc, int in64, int64_t s0, int64_t s1, int64_t s2, int64_t nitems,
                                       int64_t b0, int64_t ncx, int64_t ncy, int64_t rows_x, const void *sx,
                                       const void *sy, double *blocks, void *out, int back)
{
    const int64_t total = nitems * ncy * rows_x;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t item = e / (ncy * rows_x), r = e - item * ncy * rows_x;
        const int64_t cj = r / rows_x, ci = r - cj * rows_x;
        const int64_t b = b0 + item;
        double sc = 1.0;
        if (sx) sc *= in64 ? reinterpret_cast<const double *>(sx)[b] : (double)reinterpret_cast<const float *>(sx)[b];
        if (sy) sc *= in64 ? reinterpret_cast<const double *>(sy)[b] : (double)reinterpret_cast<const float *>(sy)[b];
        const int64_t off = b * s0 + ci * s1 + cj * s2;
        if (!back) {
            double v = 0.0;
            if (ci < ncx)
                v = in64 ? reinterpret_cast<const double *>(inc)[off] : (double)reinterpret_cast<const float *>(inc)[off];
            blocks[e] = v * sc;
        } else if (ci < ncx) {
            const double v = blocks[e] * sc;
            if (in64)
                reinterpret_cast<double *>(out)[off] = v;
            else
                reinterpret_cast<float *>(out)[off] = (float)v;
        }
    }
}

// Gradients with respect to the x side's scaled-difference rows: for each
// matrix row m (x path il, cell ci), part[slice][m][k] = sum over the slice's
// y cells n paired with it (Gram: all of them; pairwise: its own pair's) of
// G[n][m] * dyt[n][k].  grad_points_kernel adds the slices in order.
// dxt / dyt are the scaled differences in row layout (one row of d values per
// cell; x rows padded to rows_x per path with zeros), so that the inner loops
// index them directly.
struct GradContractParams {
    int op;
    const double *mat;     // dk/dc
    int64_t ld, rows_x, ncx, ncy;
    int64_t nrows_m;       // Gram: ld; pairwise: nitems * rows_x
    int64_t ncols_n;       // Gram: ny * ncy; pairwise: ncy (per pair)
    const double *dxt;     // pairwise: x differences, rows m of the chunk: [m][k]
    const double *dxk;     // Gram: the same, dimension-major: [k][m] (leading dimension ld)
    const double *dyt;     // y differences, all y cells: [y path * ncy + cj][k]
    int64_t d;
    double *part;          // gx: [slice][nrows_m][d], gy of a Gram: [range of m][ncols_n][d] partial sums
    int64_t slice;         // gx: columns per slice
    int64_t mslice;        // gy of a Gram: m per range (a multiple of kGyTile)
    double *gdy;           // gy of pairs: (ny, ncy, d)
    int64_t x0;
};

// Scaled differences src[(path * d + k) * nc + r] with `rows` rows a path
// (0 for nc <= r < rows): row layout dst[(path * rows + r) * d + k], or
// dimension-major over all paths, dst[k * (npaths * rows) + path * rows + r].
template <int V = 0> // instantiated once, in kernels_grad.cu
__global__ void grad_rows_kernel(const double *src, int64_t npaths, int64_t nc, int64_t rows, int64_t d, int dim_major,
                                 double *dst)
{
    const int64_t total = npaths * rows * d;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        int64_t path, r, k;
        if (dim_major) {
            k = e / (npaths * rows);
            const int64_t rem = e - k * npaths * rows;
            path = rem / rows;
            r = rem - path * rows;
        } else {
            path = e / (rows * d);
            const int64_t rem = e - path * rows * d;
            r = rem / d;
            k = rem - r * d;
        }
        dst[e] = r < nc ? src[(path * d + k) * nc + r] : 0.0;
    }
}

// pairwise
template <int V = 0> // instantiated once, in kernels_grad.cu
__global__ void grad_gx_kernel(GradContractParams p)
{
    const int64_t mm = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (mm >= p.nrows_m) return;
    const int64_t n0 = (int64_t)blockIdx.y * p.slice;
    const int64_t n1 = n0 + p.slice < p.ncols_n ? n0 + p.slice : p.ncols_n;
    const int64_t item = mm / p.rows_x, ci = mm - item * p.rows_x;
    const double *col = p.mat + item * p.ncy * p.rows_x + ci;  // G[n][mm] = col[n * rows_x]
    const double *dyt = p.dyt + (p.x0 + item) * p.ncy * p.d;   // the pair's own y path, [n][k]
    double *out = p.part + ((int64_t)blockIdx.y * p.nrows_m + mm) * p.d;
    for (int64_t k0 = 0; k0 < p.d; k0 += 8) {
        double acc[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] = 0.0;
        const double *yk = dyt + k0;
        for (int64_t n = n0; n < n1; ++n) {
            const double gv = col[n * p.rows_x];
            const double *yn = yk + n * p.d;
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (k0 + k < p.d) acc[k] = fma(gv, yn[k], acc[k]);
        }
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (k0 + k < p.d) out[k0 + k] = acc[k];
    }
}

// Gram: a tall, skinny product that should cost one read of G.  A thread owns
// two neighbouring rows m (16-byte loads) and 8 dimensions; the y rows of a
// tile sit in shared memory, read by the whole warp at one address.  The loads
// of 8 columns are issued together: with one in flight the kernel waited 28
// issue slots per instruction on them.
constexpr int kGxThreads = 128;
constexpr int kGxTile = 64; // y cells staged at a time

template <int V = 0> // instantiated once, in kernels_grad.cu
__global__ void __launch_bounds__(kGxThreads) grad_gx_gram_kernel(GradContractParams p)
{
    __shared__ double2 ys[kGxTile][4];
    const int64_t mm = 2 * ((int64_t)blockIdx.x * kGxThreads + threadIdx.x);
    const bool own = mm < p.nrows_m;
    const int64_t n0 = (int64_t)blockIdx.y * p.slice;
    const int64_t n1 = n0 + p.slice < p.ncols_n ? n0 + p.slice : p.ncols_n;
    const double *col = p.mat + (own ? mm : 0);
    double *out = p.part + ((int64_t)blockIdx.y * p.nrows_m + mm) * p.d;
    for (int64_t k0 = 0; k0 < p.d; k0 += 8) {
        const int kn = (int)(p.d - k0 < 8 ? p.d - k0 : 8);
        double2 acc[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] = make_double2(0.0, 0.0);
        for (int64_t nt = n0; nt < n1; nt += kGxTile) {
            __syncthreads();
            for (int e = threadIdx.x; e < kGxTile * 8; e += kGxThreads) {
                const int j = e >> 3, k = e & 7;
                reinterpret_cast<double *>(ys)[e] = nt + j < n1 && k < kn ? p.dyt[(nt + j) * p.d + k0 + k] : 0.0;
            }
            __syncthreads();
            const int cnt = (int)(n1 - nt < kGxTile ? n1 - nt : kGxTile);
            const double *g = col + nt * p.ld;
            for (int j0 = 0; j0 < cnt; j0 += 8) {
                double2 gv[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) { // columns beyond the slice: 0
                    gv[j] = make_double2(0.0, 0.0);
                    if (j0 + j < cnt) gv[j] = *reinterpret_cast<const double2 *>(g + (j0 + j) * p.ld);
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const double2 y = ys[j0 + j][k];
                        acc[2 * k].x = fma(gv[j].x, y.x, acc[2 * k].x);
                        acc[2 * k].y = fma(gv[j].y, y.x, acc[2 * k].y);
                        acc[2 * k + 1].x = fma(gv[j].x, y.y, acc[2 * k + 1].x);
                        acc[2 * k + 1].y = fma(gv[j].y, y.y, acc[2 * k + 1].y);
                    }
                }
            }
        }
        if (own) {
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (k < kn) {
                    out[k0 + k] = acc[k].x;
                    out[p.d + k0 + k] = acc[k].y;
                }
        }
    }
}

// pairwise gy: one warp per y cell n = pair * ncy + cj, lanes over the pair's x cells.
template <int V = 0> // instantiated once, in kernels_grad.cu
__global__ void grad_gy_kernel(GradContractParams p)
{
    const int lane = threadIdx.x & 31;
    const int64_t n = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (n >= (p.nrows_m / p.rows_x) * p.ncy) return;
    const int64_t item = n / p.ncy, cj = n - item * p.ncy;
    const double *row = p.mat + item * p.ncy * p.rows_x + cj * p.rows_x;
    const double *xt = p.dxt + item * p.rows_x * p.d;
    const int64_t yrow = (p.x0 + item) * p.ncy + cj;
    for (int64_t k0 = 0; k0 < p.d; k0 += 8) {
        double acc[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] = 0.0;
        for (int64_t mm = lane; mm < p.rows_x; mm += 32) {
            const double gv = row[mm]; // padding rows hold 0, as do their differences
            const double *xm = xt + mm * p.d + k0;
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (k0 + k < p.d) acc[k] = fma(gv, xm[k], acc[k]);
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            double v = acc[k];
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(kFullMask, v, off);
            if (lane == 0 && k0 + k < p.d) p.gdy[yrow * p.d + k0 + k] = v;
        }
    }
}

// gy for the Gram: partial sums over a range of m of G[n][m] dx[m][k], n over all
// y cells, m over the chunk's x cells, k < d, again one read of G.  A warp owns
// kGyRows rows and 8 dimensions; its lanes take two neighbouring m each (16-byte
// loads, the next ones in flight), the differences of a tile of m come from
// shared memory (dimension-major [k][m], two tiles), and the lanes' sums meet in
// a fixed shuffle tree.  grad_points_kernel adds the ranges of m in order, in a
// call of several chunks of x paths grad_gy_reduce_kernel first.
// (One fma per shared-memory load, or the differences read from the L2 by each
// warp, cost 2.39 and 1.76 ms for the 2.1 GB of a 128 x 128 gradient.)
constexpr int kGyRows = 8;
constexpr int kGyWarps = 4;
constexpr int kGyTile = 128; // m per tile

template <int V = 0> // instantiated once, in kernels_grad.cu
__global__ void __launch_bounds__(kGyWarps * 32, 2) grad_gy_gram_kernel(GradContractParams p)
{
    __shared__ __align__(16) double xs[2][8][kGyTile];
    const int lane = threadIdx.x & 31;
    const int64_t n0 = ((int64_t)blockIdx.x * kGyWarps + (threadIdx.x >> 5)) * kGyRows;
    const int64_t mb = (int64_t)blockIdx.y * p.mslice;
    const int64_t me = mb + p.mslice < p.ld ? mb + p.mslice : p.ld; // both multiples of 4
    const double *row[kGyRows];
#pragma unroll
    for (int r = 0; r < kGyRows; ++r) // rows beyond the last repeat it (not written)
        row[r] = p.mat + (n0 + r < p.ncols_n ? n0 + r : p.ncols_n - 1) * p.ld;
    auto load_g = [&](int64_t m, double2 (&v)[kGyRows]) {
#pragma unroll
        for (int r = 0; r < kGyRows; ++r) {
            v[r] = make_double2(0.0, 0.0);
            if (m < me) v[r] = *reinterpret_cast<const double2 *>(row[r] + m);
        }
    };
    for (int64_t k0 = 0; k0 < p.d; k0 += 8) {
        const int kn = (int)(p.d - k0 < 8 ? p.d - k0 : 8);
        auto stage = [&](int64_t m0, int buf) {
            for (int e = threadIdx.x; e < 8 * kGyTile / 2; e += kGyWarps * 32) {
                const int k = e / (kGyTile / 2), i = 2 * (e - k * (kGyTile / 2));
                const bool in = k < kn && m0 + i < me;
                grad_cp_async16z(&xs[buf][k][i], in ? p.dxk + (k0 + k) * p.ld + m0 + i : p.dxk, in ? 16 : 0);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        double acc[kGyRows][8];
#pragma unroll
        for (int r = 0; r < kGyRows; ++r)
#pragma unroll
            for (int k = 0; k < 8; ++k) acc[r][k] = 0.0;
        double2 gn[kGyRows];
        load_g(mb + 2 * lane, gn);
        __syncthreads(); // the previous dimensions are done with the tiles
        stage(mb, 0);
        int buf = 0;
        for (int64_t m0 = mb; m0 < me; m0 += kGyTile, buf ^= 1) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads(); // this tile is visible; the other is free
            if (m0 + kGyTile < me) stage(m0 + kGyTile, buf ^ 1);
#pragma unroll
            for (int h = 0; h < kGyTile / 64; ++h) {
                double2 g[kGyRows];
#pragma unroll
                for (int r = 0; r < kGyRows; ++r) g[r] = gn[r];
                load_g(m0 + 64 * (h + 1) + 2 * lane, gn);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const double2 x = *reinterpret_cast<const double2 *>(&xs[buf][k][64 * h + 2 * lane]);
#pragma unroll
                    for (int r = 0; r < kGyRows; ++r) acc[r][k] = fma(g[r].y, x.y, fma(g[r].x, x.x, acc[r][k]));
                }
            }
        }
#pragma unroll
        for (int r = 0; r < kGyRows; ++r)
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                double v = acc[r][k];
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(kFullMask, v, off);
                if (lane == 0 && k < kn && n0 + r < p.ncols_n)
                    p.part[((int64_t)blockIdx.y * p.ncols_n + n0 + r) * p.d + k0 + k] = v;
            }
    }
}

// gdy[e] (first: =, else +=) the sum over the ranges of m of part[range][e], in order: Grams of several chunks.
template <int V = 0> // instantiated once, in kernels_grad.cu
__global__ void grad_gy_reduce_kernel(const double *part, int64_t nranges, int64_t total, int first, double *gdy)
{
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= total) return;
    double s = 0.0;
    for (int64_t i = 0; i < nranges; ++i) s += part[i * total + e];
    gdy[e] = first ? s : gdy[e] + s;
}

// Gradient at the points of paths path0, ..: g[path][t][k] = scale(path) * (gd[t-1][k] - gd[t][k]), gd of the
// path's coarse differences, each the sum over nparts partial sums in order, in the output dtype.  A path has
// `pitch` rows of d values in a partial sum, which is `stride` values long.  The sums are formed here, twice a
// cell, rather than by a launch before this one: on a small batch the launch costs more.
template <int V = 0> // instantiated once, in kernels_grad.cu
__global__ void grad_points_kernel(const double *part, int64_t nparts, int64_t stride, int64_t pitch, int64_t path0,
                                   int64_t npaths, int64_t len, int64_t d, double f, const void *sc, int in64,
                                   void *out)
{
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= npaths * len * d) return;
    const int64_t pth = e / (len * d), r = e - pth * len * d, t = r / d, k = r - t * d;
    const int64_t nc = len - 1;
    const double *g = part + (pth * pitch + t) * d + k;
    double a = 0.0, b = 0.0;
    for (int64_t i = 0; i < nparts; ++i) {
        if (t >= 1) a += g[i * stride - d];
        if (t < nc) b += g[i * stride];
    }
    const double s = sc ? (in64 ? reinterpret_cast<const double *>(sc)[path0 + pth]
                                : (double)reinterpret_cast<const float *>(sc)[path0 + pth]) : 1.0;
    const double v = (a - b) * f * s;
    if (in64)
        reinterpret_cast<double *>(out)[path0 * len * d + e] = v;
    else
        reinterpret_cast<float *>(out)[path0 * len * d + e] = (float)v;
}

// All layouts of the scaled differences that a backward pass reads, straight from the points in one launch: x and y
// dimension-major per path (as delta_kernel), y by cells, and, where the pairs are one chunk, x as grad_rows_kernel.
struct GradStageParams {
    const void *x, *y, *sx, *sy;
    double fx;                    // static scale * 4^-order, on the x side
    int64_t nx, ny, ncx, ncy, d;
    double *dx, *dy, *dyt, *dxt;  // dxt may be null
    int64_t rows_x;
    int dim_major;                // dxt: [k][path * rows_x + r], else [path * rows_x + r][k]
};

template <typename TIN>
__device__ __forceinline__ double grad_diff(const void *x_, const void *s_, double f, int64_t nc, int64_t d,
                                            int64_t path, int64_t c, int64_t k)
{
    const TIN *x = reinterpret_cast<const TIN *>(x_) + (path * (nc + 1) + c) * d + k;
    const double g = s_ ? f * (double)reinterpret_cast<const TIN *>(s_)[path] : f;
    return ((double)x[d] - (double)x[0]) * g;
}

template <typename TIN>
__global__ void grad_stage_kernel(GradStageParams p)
{
    const int64_t tx = p.nx * p.ncx * p.d, ty = p.ny * p.ncy * p.d, txt = p.dxt ? p.nx * p.rows_x * p.d : 0;
    const int64_t total = tx + 2 * ty + txt;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        int64_t e = i;
        if (e < tx) {
            const int64_t row = e / p.ncx, c = e - row * p.ncx, path = row / p.d, k = row - path * p.d;
            p.dx[e] = grad_diff<TIN>(p.x, p.sx, p.fx, p.ncx, p.d, path, c, k);
            continue;
        }
        e -= tx;
        if (e < ty) {
            const int64_t row = e / p.ncy, c = e - row * p.ncy, path = row / p.d, k = row - path * p.d;
            p.dy[e] = grad_diff<TIN>(p.y, p.sy, 1.0, p.ncy, p.d, path, c, k);
            continue;
        }
        e -= ty;
        if (e < ty) {
            const int64_t row = e / p.d, k = e - row * p.d, path = row / p.ncy, c = row - path * p.ncy;
            p.dyt[e] = grad_diff<TIN>(p.y, p.sy, 1.0, p.ncy, p.d, path, c, k);
            continue;
        }
        e -= ty;
        int64_t row, k;
        if (p.dim_major) {
            k = e / (p.nx * p.rows_x);
            row = e - k * p.nx * p.rows_x;
        } else {
            row = e / p.d;
            k = e - row * p.d;
        }
        const int64_t path = row / p.rows_x, c = row - path * p.rows_x;
        p.dxt[e] = c < p.ncx ? grad_diff<TIN>(p.x, p.sx, p.fx, p.ncx, p.d, path, c, k) : 0.0;
    }
}

} // namespace sigk
