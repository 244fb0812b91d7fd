// Two-pass symmetry-function kernels, FP32 (mixed forms).
#include "sf_pair_launch.cuh"

namespace n2p2b
{

N2P2B_PAIR_LAUNCH(anyallf, float, -1, 5, (sfp2::kHasPow2 | sfp2::kHasLadder | sfp2::kHasGeneral
                   | sfp2::kHasCompact), 4, 4)

} // namespace n2p2b
