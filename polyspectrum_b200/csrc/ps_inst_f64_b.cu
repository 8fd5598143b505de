// Pass kernels, FP64, 320 and 384 points (see ps_launch.cuh).
#include "ps_launch_impl.cuh"

namespace ps {
PS_INSTANTIATE_L3_B(double)
}  // namespace ps
