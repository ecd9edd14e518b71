// Predictive local systems (local_warp.cuh).
#include "local_warp_launch.cuh"

namespace nngp {
template nngp_status launch_predict<float>(const LocalArgs &, const float *, const float *, const float *,
                                           const int32_t *, float *, float *, int32_t *, cudaStream_t);
template nngp_status launch_predict<double>(const LocalArgs &, const double *, const double *, const double *,
                                            const int32_t *, double *, double *, int32_t *, cudaStream_t);
}  // namespace nngp
