// Instantiations of norm_warp_kernel.
#include "dispatch.h"
#include "norm_warp.cuh"

namespace sigk {
namespace {
template <typename TIN, int R, int M>
NormFn by_o(int O)
{
    switch (O) {
    case 0: return norm_warp_kernel<TIN, R, 0, M>;
    case 1: return norm_warp_kernel<TIN, R, 1, M>;
    case 2: return norm_warp_kernel<TIN, R, 2, M>;
    case 3: return norm_warp_kernel<TIN, R, 3, M>;
    default: return norm_warp_kernel<TIN, R, 4, M>;
    }
}
template <typename TIN, int M>
NormFn by_r(int R, int O)
{
    switch (R) {
    case 2: return by_o<TIN, 2, M>(O);
    case 4: return by_o<TIN, 4, M>(O);
    case 8: return by_o<TIN, 8, M>(O);
    default: return by_o<TIN, 16, M>(O);
    }
}
} // namespace

NormFn get_norm_warp_kernel(bool in64, int mode, int R, int O)
{
    switch (mode) {
    case kNormGiven: return in64 ? by_r<double, kNormGiven>(R, O) : by_r<float, kNormGiven>(R, O);
    case kNormTile: return by_r<double, kNormTile>(R, O);
    default: return by_r<double, kNormDelta>(R, O);
    }
}
} // namespace sigk
