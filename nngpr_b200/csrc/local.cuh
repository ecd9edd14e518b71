// Shared pieces of the local-systems kernels (local.cu, local_warp.cuh): arguments, kernel functions.
#pragma once

#include <cmath>
#include <type_traits>

#include "common.cuh"

namespace nngp {

constexpr int kMaxDimLocal = 256;
constexpr int kMaxTheta = kMaxDimLocal + 3;
constexpr int kWarpM = 64;  // neighbours of the warp kernel
constexpr int kRedoM = 32;  // up to here FP32 inputs are solved in FP32 (FP64 re-solves), above in FP64
constexpr double kHalfLog2Pi = 0.91893853320467274178;

struct LocalArgs {
    double rbf, cst, noise, alpha;
    double pivot_abs;  // FP32 systems with a pivot below this are re-solved in FP64
    int64_t n_rows;    // rows of x_ref / y_ref (neighbour index bound)
    int64_t n_points;
    int d, ydim, m;
    int ard;  // 1: per-feature length scales
    int family;  // stationary part: NNGP_FAMILY_RBF or a Matern (include/nngp_b200.h)
    int64_t alpha_below;  // alpha goes on the diagonal slots of neighbours with index < alpha_below
    int weights_out;      // predict: write w = K_nn^-1 k (a.m per point) to `mean` instead of the mean
    int idx_rbf, idx_const, idx_noise, idx_ls, n_theta;
    unsigned long long *fp64_count;  // systems re-solved in FP64 are added here (may be null)
    // fit step with FP32 inputs: bit p marks point p (counted from the launch's first row), whose
    // FP32 system needs the FP64 re-solve that local_redo_kernel then runs (predict re-solves in
    // place and leaves this null)
    uint32_t *redo_bits;
    // device block of nngp_theta_params (may be null): [rbf, cst, noise, pivot_abs, 1/l_f ...];
    // when set, the kernels take these values instead of the fields above
    const double *dev_params;
    double inv_ls[kMaxDimLocal];
};

// The hyperparameter values a kernel works with: from the arguments, or from the device block
// of a theta that never left the device.
struct Hyp {
    double rbf, cst, noise, pivot_abs;
    const double *inv_ls;
};
__device__ __forceinline__ Hyp hyp_of(const LocalArgs &a) {
    if (a.dev_params) {
        const double *q = a.dev_params;
        return Hyp{q[0], q[1], q[2], q[3], q + 4};
    }
    return Hyp{a.rbf, a.cst, a.noise, a.pivot_abs, a.inv_ls};
}

template <typename T> __device__ __forceinline__ T dsqrt(T v) { return sqrt(v); }
template <typename T> __device__ __forceinline__ T drsqrt(T v) { return rsqrt(v); }
template <> __device__ __forceinline__ float drsqrt<float>(float v) { return rsqrtf(v); }

// e^x for x <= 0 without a branch, so that the exponentials of several entries run interleaved
// (exp() has a slow path, and its branch kept the entries of a lane one after the other).
// FP64: x = n ln 2 + r, |r| <= ln(2) / 2 (Cody and Waite's two-part reduction), e^r = 1 + r + r^2 q(r) with q the
// degree-9 interpolant of (e^r - 1 - r) / r^2 at the Chebyshev nodes (error 1.7e-17), times 2^n.  At most 0.85 ulp
// off over 6e7 arguments in [-700, 0]; below -708 (results under 3e-308) it is 0; NaN stays NaN.
__device__ __forceinline__ float exp_neg(float x) { return expf(x); }
__device__ __forceinline__ double exp_neg(double x) {
    const double t = fma(x, 0x1.71547652b82fep+0, 0x1.8p52);  // the integer n in the low word
    const double n = t - 0x1.8p52;
    double r = fma(n, -0x1.62e42fefap-1, x);
    r = fma(n, -0x1.cf79abc9e3b3ap-40, r);
    double q = 0x1.af38d53857513p-26;
    q = fma(q, r, 0x1.2891a8c1d838dp-22);
    q = fma(q, r, 0x1.71de0d9c145d0p-19);
    q = fma(q, r, 0x1.a019b8ef67c6cp-16);
    q = fma(q, r, 0x1.a01a01a7c8d47p-13);
    q = fma(q, r, 0x1.6c16c17893833p-10);
    q = fma(q, r, 0x1.11111111109adp-7);
    q = fma(q, r, 0x1.5555555553d4fp-5);
    q = fma(q, r, 0x1.5555555555556p-3);
    q = fma(q, r, 0x1.0000000000001p-1);
    const double a = 1.0 + r, b = (1.0 - a) + r;  // a + b = 1 + r exactly
    const double p = a + fma(q, r * r, b);
    const double s = __hiloint2double((1023 + __double2loint(t)) << 20, 0);
    return x < -708.0 ? 0.0 : p * s;
}

// Unit-amplitude stationary part s of the kernel at squared scaled distance sq (formulas of
// nngpr/batched_kernels.py:1070-1088 for the Matern kernels; RBF exp(-sq / 2)).
template <bool MATERN, typename T> __device__ __forceinline__ T kern_s(int family, T sq) {
    if (!MATERN || family == NNGP_FAMILY_RBF) return exp_neg(T(-0.5) * sq);
    if (family == NNGP_FAMILY_MATERN12) return exp_neg(-dsqrt<T>(sq));
    if (family == NNGP_FAMILY_MATERN32) {
        const T r = dsqrt<T>(T(3) * sq);
        return (T(1) + r) * exp_neg(-r);
    }
    const T r = dsqrt<T>(T(5) * sq);
    return (T(1) + r + r * r / T(3)) * exp_neg(-r);
}

// g with d s / d log l_f = g * t_f^2 (t_f the scaled difference of feature f); isotropic:
// d s / d log l = g * sq.  `s` is kern_s at the same sq.  Reference gradients:
// nngpr/batched_kernels.py:1108-1120 (Matern), :895-898 (RBF).
template <bool MATERN, typename T> __device__ __forceinline__ T kern_g(int family, T sq, T s) {
    if (!MATERN || family == NNGP_FAMILY_RBF) return s;
    if (family == NNGP_FAMILY_MATERN12) {
        const T r = dsqrt<T>(sq);
        return r > T(0) ? s / r : T(0);  // every t_f is 0 where r is
    }
    if (family == NNGP_FAMILY_MATERN32) return T(3) * exp_neg(-dsqrt<T>(T(3) * sq));
    const T r = dsqrt<T>(T(5) * sq);
    return T(5) / T(3) * (T(1) + r) * exp_neg(-r);
}

}  // namespace nngp
