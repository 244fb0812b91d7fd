// Two-pass symmetry-function kernels, FP64 (plain form).
#include "sf_pair_launch.cuh"

namespace n2p2b
{

N2P2B_PAIR_LAUNCH(anyall, double, -1, 5, (sfp2::kHasPow2 | sfp2::kHasLadder | sfp2::kHasGeneral
                   | sfp2::kHasCompact), 3, 3)

} // namespace n2p2b
