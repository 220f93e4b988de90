// Instantiations of pair_wave_kernel.
#include "dispatch.h"
#include "pair_wave.cuh"

namespace sigk {
namespace {
template <int R, int O>
PairWaveKernel shape()
{
    using NS = NormShape<R, O>;
    return {pair_wave_kernel<R, O>, NS::C, NS::RC, NS::CC, NS::MAXW};
}
template <int R>
PairWaveKernel by_o(int O)
{
    switch (O) {
    case 0:
        if constexpr (R <= 4) return shape<R, 0>();
        return PairWaveKernel{};
    case 1: return shape<R, 1>();
    case 2: return shape<R, 2>();
    case 3: return shape<R, 3>();
    default: return shape<R, 4>();
    }
}
} // namespace

PairWaveKernel get_pair_wave_kernel(int R, int O)
{
    switch (R) {
    case 2: return by_o<2>(O);
    case 4: return by_o<4>(O);
    case 8: return by_o<8>(O);
    default: return PairWaveKernel{};
    }
}
} // namespace sigk
