// Pass kernels, FP32, 512 and 1024 points (see ps_launch.cuh).
#include "ps_launch_impl.cuh"

namespace ps {
PS_INSTANTIATE_L3_C(float)
}  // namespace ps
