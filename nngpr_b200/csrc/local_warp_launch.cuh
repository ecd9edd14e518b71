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
    const int M = warp_rows(a.m), C = rows_per_lane(M, a.d, a.n_points, F32, false);
    auto pick = [&](auto rows, auto per_lane) {
        constexpr int R = decltype(rows)::value, P = decltype(per_lane)::value;
        return rbf ? (grad ? local_warp_kernel<TIn, R, P, true, false, false>
                           : local_warp_kernel<TIn, R, P, false, false, false>)
                   : (grad ? local_warp_kernel<TIn, R, P, true, false, true>
                           : local_warp_kernel<TIn, R, P, false, false, true>);
    };
    using I1 = std::integral_constant<int, 1>;
    using I2 = std::integral_constant<int, 2>;
    auto pick_rows = [&](auto rows) { return C == 1 ? pick(rows, I1{}) : pick(rows, I2{}); };
    auto fn = M == 16   ? pick_rows(std::integral_constant<int, 16>{})
              : M == 32 ? pick_rows(std::integral_constant<int, 32>{})
                        : pick(std::integral_constant<int, 64>{}, I2{});
    const int groups = 32 / lanes_per_point(M, C);
    const bool keep_e = grad && rbf && M <= 32;
    const size_t bytes = (F32 && M <= 32 ? WarpLayout::make<true, false>(M, C, a.d, a.n_theta, grad, keep_e, grad && a.ard)
                                         : WarpLayout::make<false, true>(M, C, a.d, a.n_theta, grad, keep_e, grad && a.ard))
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
    const int M = warp_rows(a.m), C = rows_per_lane(M, a.d, a.n_points, F32, true);
    auto pick = [&](auto rows, auto per_lane) {
        constexpr int R = decltype(rows)::value, P = decltype(per_lane)::value;
        return rbf ? local_warp_kernel<TIn, R, P, false, true, false> : local_warp_kernel<TIn, R, P, false, true, true>;
    };
    using I1 = std::integral_constant<int, 1>;
    using I2 = std::integral_constant<int, 2>;
    auto pick_rows = [&](auto rows) { return C == 1 ? pick(rows, I1{}) : pick(rows, I2{}); };
    auto fn = M == 16   ? pick_rows(std::integral_constant<int, 16>{})
              : M == 32 ? pick_rows(std::integral_constant<int, 32>{})
                        : pick(std::integral_constant<int, 64>{}, I2{});
    const int groups = 32 / lanes_per_point(M, C);
    const size_t bytes = (F32 && M <= 32 ? WarpLayout::make<true, true>(M, C, a.d, 0, false, false, false)
                                         : WarpLayout::make<false, true>(M, C, a.d, 0, false, false, false))
                             .total;
    WarpLaunch w;
    nngp_status st = warp_launch(reinterpret_cast<const void *>(fn), bytes, (a.n_points + groups - 1) / groups, 0, &w);
    if (st != NNGP_OK) return st;
    fn<<<w.grid, w.warps * 32, w.smem, stream>>>(a, x_ref, y_ref, x_pt, nullptr, nbr, nullptr, mean, var, flags);
    NNGP_CUDA_TRY(cudaGetLastError());
    return NNGP_OK;
}

}  // namespace nngp
