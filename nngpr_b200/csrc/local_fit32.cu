// Fit-step local systems of FP32 inputs (local_warp.cuh).
#include "local_warp_launch.cuh"

namespace nngp {
template nngp_status launch_fit<float>(const LocalArgs &, bool, const float *, const float *, const float *,
                                       const float *, const int32_t *, double *, int, int *, int32_t *, cudaStream_t);
}  // namespace nngp
