// Launchers of the kernels of local_warp.cuh (instantiated in local_fit32.cu, local_fit64.cu and
// local_pred.cu).
#pragma once

#include "local_warp.cuh"

namespace nngp {

template <typename TIn>
nngp_status launch_fit(const LocalArgs &a, bool grad, const TIn *x_ref, const TIn *y_ref, const TIn *x_pt,
                       const TIn *y_pt, const int32_t *nbr, double *block_out, int grid_limit, int *parts,
                       int32_t *flags, cudaStream_t stream) {
    constexpr bool F32 = std::is_same<TIn, float>::value;
    const bool rbf = a.family == NNGP_FAMILY_RBF;
    const int M = warp_rows(a.m);
    auto pick = [&](auto rows) {
        constexpr int R = decltype(rows)::value;
        return rbf ? (grad ? local_warp_kernel<TIn, R, true, false, false> : local_warp_kernel<TIn, R, false, false, false>)
                   : (grad ? local_warp_kernel<TIn, R, true, false, true> : local_warp_kernel<TIn, R, false, false, true>);
    };
    auto fn = M == 16   ? pick(std::integral_constant<int, 16>{})
              : M == 32 ? pick(std::integral_constant<int, 32>{})
                        : pick(std::integral_constant<int, 64>{});
    const int groups = 32 / lanes_per_point(M);
    const bool keep_e = grad && rbf && M <= 32;
    const size_t bytes = (F32 && M <= 32 ? WarpLayout::make<true, false>(M, a.d, a.n_theta, grad, keep_e, grad && a.ard)
                                         : WarpLayout::make<false, true>(M, a.d, a.n_theta, grad, keep_e, grad && a.ard))
                             .total;
    WarpLaunch w;
    nngp_status st = warp_launch(reinterpret_cast<const void *>(fn), bytes, (a.n_points + groups - 1) / groups,
                                 grid_limit, &w);
    if (st != NNGP_OK) return st;
    fn<<<w.grid, w.warps * 32, w.smem, stream>>>(a, x_ref, y_ref, x_pt, y_pt, nbr, block_out, nullptr, nullptr, flags);
    NNGP_CUDA_TRY(cudaGetLastError());
    *parts = w.grid;
    return NNGP_OK;
}

template <typename TIn>
nngp_status launch_predict(const LocalArgs &a, const TIn *x_ref, const TIn *y_ref, const TIn *x_pt,
                           const int32_t *nbr, TIn *mean, TIn *var, int32_t *flags, cudaStream_t stream) {
    constexpr bool F32 = std::is_same<TIn, float>::value;
    const bool rbf = a.family == NNGP_FAMILY_RBF;
    const int M = warp_rows(a.m);
    auto pick = [&](auto rows) {
        constexpr int R = decltype(rows)::value;
        return rbf ? local_warp_kernel<TIn, R, false, true, false> : local_warp_kernel<TIn, R, false, true, true>;
    };
    auto fn = M == 16   ? pick(std::integral_constant<int, 16>{})
              : M == 32 ? pick(std::integral_constant<int, 32>{})
                        : pick(std::integral_constant<int, 64>{});
    const int groups = 32 / lanes_per_point(M);
    const size_t bytes = (F32 && M <= 32 ? WarpLayout::make<true, true>(M, a.d, 0, false, false, false)
                                         : WarpLayout::make<false, true>(M, a.d, 0, false, false, false))
                             .total;
    WarpLaunch w;
    nngp_status st = warp_launch(reinterpret_cast<const void *>(fn), bytes, (a.n_points + groups - 1) / groups, 0, &w);
    if (st != NNGP_OK) return st;
    fn<<<w.grid, w.warps * 32, w.smem, stream>>>(a, x_ref, y_ref, x_pt, nullptr, nbr, nullptr, mean, var, flags);
    NNGP_CUDA_TRY(cudaGetLastError());
    return NNGP_OK;
}

}  // namespace nngp
