// Instantiations of the backward-pass kernels (grad.cuh).
#include "dispatch.h"
#include "grad.cuh"

namespace sigk {
namespace {
template <int R, int O, int W>
GradFns grad_fns()
{
    using GS = GradShape<R, O, W>;
    return {grad_fwd_kernel<R, O, W>, grad_bwd_kernel<R, O, W>, GS::C, GS::CC, GS::CTAS, GS::REC,
            grad_bwd_smem<R, O, W>()};
}
template <int R, int W>
GradFns grad_by_o(int O)
{
    switch (O) {
    case 0:
        if constexpr (R <= 4 && W == 1) return grad_fns<R, 0, W>();
        return GradFns{};
    case 1:
        if constexpr (R <= 4) return grad_fns<R, 1, W>();
        return GradFns{};
    case 2:
        if constexpr (R >= 4 && R <= 8) return grad_fns<R, 2, W>();
        return GradFns{};
    case 3:
        if constexpr (R == 8) return grad_fns<R, 3, W>();
        return GradFns{};
    case 4:
        if constexpr (R == 16 && W == 1) return grad_fns<R, 4, W>();
        return GradFns{};
    default: return GradFns{};
    }
}
template <int W>
GradFns grad_by_r(int R, int O)
{
    switch (R) {
    case 2: return grad_by_o<2, W>(O);
    case 4: return grad_by_o<4, W>(O);
    case 8: return grad_by_o<8, W>(O);
    case 16: return grad_by_o<16, W>(O);
    default: return GradFns{};
    }
}
} // namespace

GradFns get_grad_kernels(int R, int O, bool wide) { return wide ? grad_by_r<2>(R, O) : grad_by_r<1>(R, O); }

GradAuxFns get_grad_aux_kernels()
{
    return {grad_pair_inc_kernel<>, grad_gx_kernel<>, grad_gy_kernel<>, grad_points_kernel<>,
            grad_stage_kernel<float>, grad_stage_kernel<double>, grad_rows_kernel<>, grad_gx_gram_kernel<>,
            grad_gy_gram_kernel<>, grad_gy_reduce_kernel<>, grad_inc_blocks_kernel<>};
}

} // namespace sigk
