// Instantiations of the second-difference kernels.
#include "dispatch.h"
#include "second_diff.cuh"

namespace sigk {
namespace {
template <typename I>
SecondDiffFn pick(bool adjoint, bool src64, bool dst64)
{
    if (adjoint)
        return src64 ? (dst64 ? second_diff_grad_kernel<double, double, I> : second_diff_grad_kernel<double, float, I>)
                     : (dst64 ? second_diff_grad_kernel<float, double, I> : second_diff_grad_kernel<float, float, I>);
    return src64 ? (dst64 ? second_diff_kernel<double, double, I> : second_diff_kernel<double, float, I>)
                 : (dst64 ? second_diff_kernel<float, double, I> : second_diff_kernel<float, float, I>);
}
} // namespace

SecondDiffFn get_second_diff_kernel(bool adjoint, bool src64, bool dst64, bool wide)
{
    return wide ? pick<int64_t>(adjoint, src64, dst64) : pick<uint32_t>(adjoint, src64, dst64);
}

} // namespace sigk
