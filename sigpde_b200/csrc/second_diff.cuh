// second_diff.cuh -- coarse increments of static-kernel values, and their adjoint.
//
// For a static kernel the device does not know, torch evaluates G(x_i, y_j) and
// autograd continues through it; the increments
//   inc(i, j) = (G(i+1, j+1) + G(i, j) - G(i+1, j) - G(i, j+1)) / 4^order
// (sigpde/torch/kernel.py:13-21) were five torch operations on slices, and
// their backward a zero-filled copy, a negation and a sum per slice.  A training
// step on a small batch is bound by those launches and the graph nodes behind
// them, so each direction is one pass here.  Both keep the order and the type of
// the torch expressions: the sums are rounded in G's type, the adjoint adds the
// slices' shares in the order in which autograd visits them.
#pragma once

#include <cstdint>

namespace sigk {

struct SecondDiffParams {
    const void *src;   // forward: G; adjoint: dL/dinc, contiguous (pairs, rows - 1, cols - 1)
    void *dst;         // forward: inc, contiguous; adjoint: dL/dG
    int64_t na, nb;    // pairs (a, b)
    int64_t rows, cols;
    int64_t s0, s1, s2, s3; // element strides of G (adjoint: of dL/dG)
    double scale;      // 4^-order
};

// One thread an element of the result; I indexes them (32 bits where they fit:
// the three divisions are then a few instructions each).
template <typename T, typename TO, typename I>
__global__ void second_diff_kernel(SecondDiffParams p)
{
    const T *__restrict__ G = reinterpret_cast<const T *>(p.src);
    TO *__restrict__ inc = reinterpret_cast<TO *>(p.dst);
    const I nr = (I)(p.rows - 1), nc = (I)(p.cols - 1), nb = (I)p.nb;
    const I total = (I)(p.na * p.nb) * nr * nc;
    for (I e = (I)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (I)gridDim.x * blockDim.x) {
        const I row = e / nc, j = e - row * nc, pair = row / nr, i = row - pair * nr, a = pair / nb, b = pair - a * nb;
        const T *g = G + (int64_t)a * p.s0 + (int64_t)b * p.s1 + (int64_t)i * p.s2 + (int64_t)j * p.s3;
        const T v = g[p.s2 + p.s3] + g[0] - g[p.s2] - g[p.s3];
        inc[e] = TO(v * T(p.scale));
    }
}

// T: type of dL/dinc, TG: type of G
template <typename T, typename TG, typename I>
__global__ void second_diff_grad_kernel(SecondDiffParams p)
{
    const T *__restrict__ gi = reinterpret_cast<const T *>(p.src);
    TG *__restrict__ gg = reinterpret_cast<TG *>(p.dst);
    const I rows = (I)p.rows, cols = (I)p.cols, nb = (I)p.nb;
    const I total = (I)(p.na * p.nb) * rows * cols;
    for (I e = (I)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (I)gridDim.x * blockDim.x) {
        const I row = e / cols, j = e - row * cols, pair = row / rows, i = row - pair * rows, a = pair / nb,
                b = pair - a * nb;
        const T *g = gi + ((int64_t)pair * (rows - 1) + i) * (cols - 1) + j; // inc(i, j)
        const bool r0 = i > 0, r1 = i + 1 < rows, c0 = j > 0, c1 = j + 1 < cols;
        const TG sc = TG(p.scale);
        TG v = TG(0);
        if (r1 && c0) v -= TG(g[-1]) * sc;                    // as inc(i, j-1)'s G(i, j)
        if (r0 && c1) v -= TG(g[-((int64_t)cols - 1)]) * sc;  // inc(i-1, j)
        if (r1 && c1) v += TG(g[0]) * sc;                     // inc(i, j)
        if (r0 && c0) v += TG(g[-(int64_t)cols]) * sc;        // inc(i-1, j-1)
        gg[(int64_t)a * p.s0 + (int64_t)b * p.s1 + (int64_t)i * p.s2 + (int64_t)j * p.s3] = v;
    }
}

} // namespace sigk
