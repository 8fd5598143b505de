// Pass kernels, FP32, 16 to 256 points (see ps_launch.cuh).
#include "ps_launch_impl.cuh"

namespace ps {
PS_INSTANTIATE_L3_A(float)
}  // namespace ps
