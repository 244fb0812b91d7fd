// Two-pass symmetry-function kernels, FP64 (plain form).
#include "sf_pair_launch.cuh"

namespace n2p2b
{

N2P2B_PAIR_LAUNCH(poly4, double, 6, 5, (sfp2::kHasPow2), 3, 4)

} // namespace n2p2b
