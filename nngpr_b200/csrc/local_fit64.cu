// Fit-step local systems of FP64 inputs (local_warp.cuh).
#include "local_warp_launch.cuh"

namespace nngp {
template nngp_status launch_fit<double>(const LocalArgs &, bool, const double *, const double *, const double *,
                                        const double *, const int32_t *, double *, int, int *, int32_t *, cudaStream_t);
}  // namespace nngp
