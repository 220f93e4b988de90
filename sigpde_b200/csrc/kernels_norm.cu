// Instantiations of norm_kernel (float64 cells and bracket arithmetic).
#include "dispatch.h"
#include "norm_wave.cuh"

namespace sigk {
namespace {
template <int R, int O>
NormKernel by_mem(bool smem_tile, bool smem_bnd)
{
    using NS = NormShape<R, O>;
    const int regs = R == 16 ? 255 : 128;
    return {smem_tile && smem_bnd ? norm_kernel<R, O, true, true>
            : smem_bnd            ? norm_kernel<R, O, false, true>
                                  : norm_kernel<R, O, false, false>,
            NS::C, NS::RC, NS::CC,
            NS::MAXW, regs};
}
template <int R>
NormKernel by_o(int O, bool smem_tile, bool smem_bnd)
{
    switch (O) {
    case 0:
        if constexpr (R <= 4) return by_mem<R, 0>(smem_tile, smem_bnd); // 16 coarse cells a step would spill
        return NormKernel{};
    case 1: return by_mem<R, 1>(smem_tile, smem_bnd);
    case 2: return by_mem<R, 2>(smem_tile, smem_bnd);
    case 3: return by_mem<R, 3>(smem_tile, smem_bnd);
    default: return by_mem<R, 4>(smem_tile, smem_bnd);
    }
}
} // namespace

NormKernel get_norm_kernel(int R, int O, bool smem_tile, bool smem_bnd)
{
    switch (R) {
    case 2: return by_o<2>(O, smem_tile, smem_bnd);
    case 4: return by_o<4>(O, smem_tile, smem_bnd);
    case 8: return by_o<8>(O, smem_tile, smem_bnd);
    default: return by_o<16>(O, smem_tile, smem_bnd);
    }
}
} // namespace sigk
