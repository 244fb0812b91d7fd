// Two-pass symmetry-function kernels, FP32 (mixed forms).
#include "sf_pair_launch.cuh"

namespace n2p2b
{

N2P2B_PAIR_LAUNCH(any4f, float, -1, 5, (sfp2::kHasPow2), 4, 6)

} // namespace n2p2b
