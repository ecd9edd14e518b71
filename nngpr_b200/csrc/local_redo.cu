// FP64 re-solve of marked FP32 fit-step systems (local_warp.cuh).
#include "local_warp_launch.cuh"

namespace nngp {

nngp_status launch_redo(const LocalArgs &a, bool grad, const float *x_ref, const float *y_ref, const float *x_pt,
                        const float *y_pt, const int32_t *nbr, double *block_out, int grid_limit, int *parts,
                        int32_t *flags, cudaStream_t stream) {
    const bool rbf = a.family == NNGP_FAMILY_RBF;
    const int M = warp_rows(a.m);
    auto pick = [&](auto rows) {
        constexpr int R = decltype(rows)::value;
        return rbf ? (grad ? local_redo_kernel<R, true, false> : local_redo_kernel<R, false, false>)
                   : (grad ? local_redo_kernel<R, true, true> : local_redo_kernel<R, false, true>);
    };
    auto fn = M == 16 ? pick(std::integral_constant<int, 16>{}) : pick(std::integral_constant<int, 32>{});
    const size_t bytes = WarpLayout::make<false, true>(M, 2, a.d, a.n_theta, grad, grad && rbf, grad && a.ard).total;
    WarpLaunch w;
    nngp_status st = warp_launch(reinterpret_cast<const void *>(fn), bytes, (a.n_points + 31) / 32, grid_limit, &w);
    if (st != NNGP_OK) return st;
    fn<<<w.grid, w.warps * 32, w.smem, stream>>>(a, x_ref, y_ref, x_pt, y_pt, nbr, block_out, flags);
    NNGP_CUDA_TRY(cudaGetLastError());
    *parts = w.grid;
    return NNGP_OK;
}

}  // namespace nngp
