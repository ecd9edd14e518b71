// Cells of the pruned prefix search: clusters of points and separating slabs between them.
//
// In many dimensions the bounding boxes of 128 curve-neighbours meet almost every other box although the
// points themselves lie far apart: a box's diagonal grows with sqrt(d), its points' extent along one
// direction does not.  So points are also assigned to the nearest of K pivots (k-means on a sample),
// groups of rows and tiles of refs stay inside a cell, and two sets of different cells a, b are
// bounded from below along the line through their pivots: with u the unit vector from pivot a to pivot b,
//   |y - x| >= (y - x) . u = (p_b - p_a) . u - (x - p_a) . u - (y - p_b) . (-u),
// the pivots' distance less the reach of x's set towards b and of y's set towards a.  One number
// per set and pivot.  Any unit vector and any assignment give a valid bound, also for the few tiles
// that straddle two cells (measured from their first point's pivot).
//
// Rounding: u has a length of at most 1 + 2^-23 (components normalised in FP64, rounded once; u from b to a is
// the exact negative of u from a to b), which the rule that uses the slab divides out; the reach of a set is the
// FP32 maximum plus (d + 8) 2^-23 R, R >= |x - p| over the set, more than twice the error of a difference, a
// d-term FMA sum and R itself; the pivots' distance is computed in FP64 and rounded down.  NaN
// coordinates are skipped: such points are at NaN distance from everything and in no list.
//
// Measured (numpy, 100,000 points, listed pairs): 16-d mixture of 64 components 69 % with boxes, 2.1 % with 128
// cells; 8-d uniform with ARD scales 43 -> 33 %; 8-d uniform 98 -> 85 %; 5-d 28 -> 20 %.
#include <algorithm>

#include "common.cuh"
#include "knn_cells.cuh"

namespace nngp {
namespace cells {
namespace {

constexpr int kThreads = 256;
constexpr int kSample = 16384;
constexpr int kIters = 5;
constexpr int kMeansThreads = 128;
constexpr int kMaxD = 24;

int64_t sample_size(int64_t n) { return n < kSample ? n : kSample; }

// Nearest of K pivots to x (DP floats); sm4: K x DP floats, -2 x the pivot, pn: |pivot|^2.
template <int DP>
__device__ __forceinline__ int nearest(const float4 (&x)[DP / 4], const float4 *sm4, const float *pn, int K) {
    float best = pos_inf<float>();
    int bk = 0;
    for (int k = 0; k < K; ++k) {
        float s = pn[k];
#pragma unroll
        for (int v = 0; v < DP / 4; ++v) {
            const float4 q = sm4[k * (DP / 4) + v];
            s = fmaf(x[v].x, q.x, fmaf(x[v].y, q.y, fmaf(x[v].z, q.z, fmaf(x[v].w, q.w, s))));
        }
        if (s < best) {
            best = s;
            bk = k;
        }
    }
    return bk;
}

// One k-means step on the sample: the pivots of this step (step 0: every (S / K)-th sample point; else the
// means that the previous step summed, or the previous pivot where none fell to it), then each sample
// point added to the sums of its nearest pivot.  The order of the atomic additions may change a
// pivot's last bits from run to run, which never changes a list.
template <int DP>
__global__ void __launch_bounds__(kMeansThreads) kmeans_kernel(const float *__restrict__ xs, int64_t n, int d, int K,
                                                               int64_t S, int step, const float *__restrict__ prev_piv,
                                                               const float *__restrict__ prev_sum,
                                                               float *__restrict__ piv, float *__restrict__ sum,
                                                               int last) {
    extern __shared__ __align__(16) float sm[];
    float *pn = sm + K * DP;   // K: |p|^2
    float *acc = pn + K;       // K x (DP + 1)
    const int64_t stride = n / S;
    for (int e = threadIdx.x; e < K * DP; e += kMeansThreads) {
        const int k = e / DP, f = e - k * DP;
        float v;
        if (step == 0) {
            v = xs[(((int64_t)k * S / K + S / (2 * K)) * stride) * DP + f];
        } else {
            const float c = prev_sum[k * (DP + 1) + DP];
            v = c > 0.f ? prev_sum[k * (DP + 1) + f] / c : prev_piv[e];
        }
        sm[e] = -2.f * v;
        if (blockIdx.x == 0) piv[e] = v;
    }
    if (last) return;
    for (int e = threadIdx.x; e < K * (DP + 1); e += kMeansThreads) acc[e] = 0.f;
    __syncthreads();
    for (int k = threadIdx.x; k < K; k += kMeansThreads) {
        float s = 0.f;
        for (int f = 0; f < DP; ++f) s = fmaf(sm[k * DP + f], sm[k * DP + f], s);
        pn[k] = 0.25f * s;
    }
    __syncthreads();
    for (int64_t s = blockIdx.x * (int64_t)kMeansThreads + threadIdx.x; s < S; s += (int64_t)gridDim.x * kMeansThreads) {
        float4 x[DP / 4];
        bool fine = true;
#pragma unroll
        for (int v = 0; v < DP / 4; ++v) {
            x[v] = reinterpret_cast<const float4 *>(xs + s * stride * DP)[v];
            fine = fine && isfinite(x[v].x) && isfinite(x[v].y) && isfinite(x[v].z) && isfinite(x[v].w);
        }
        if (!fine) continue;
        float *to = acc + nearest<DP>(x, reinterpret_cast<const float4 *>(sm), pn, K) * (DP + 1);
#pragma unroll
        for (int v = 0; v < DP / 4; ++v) {
            atomicAdd(to + 4 * v, x[v].x);
            atomicAdd(to + 4 * v + 1, x[v].y);
            atomicAdd(to + 4 * v + 2, x[v].z);
            atomicAdd(to + 4 * v + 3, x[v].w);
        }
        atomicAdd(to + DP, 1.f);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < K * (DP + 1); e += kMeansThreads)
        if (acc[e] != 0.f) atomicAdd(sum + e, acc[e]);
}

// CTA b: the unit vectors from pivot b to every pivot a, and the pivots' distances along them.  The vector of
// the pair (a, b) is formed from the lower to the higher index, so both directions are exact negatives.
__global__ void __launch_bounds__(kMaxCells) directions_kernel(const float *__restrict__ piv, int d, int dp, int K,
                                                               float *__restrict__ dirs, float *__restrict__ apart) {
    const int b = blockIdx.x, a = threadIdx.x;
    if (a >= K) return;
    const int lo = min(a, b), hi = max(a, b);
    double len2 = 0.0;
    for (int f = 0; f < d; ++f) {
        const double t = (double)piv[hi * dp + f] - (double)piv[lo * dp + f];
        len2 = fma(t, t, len2);
    }
    const double inv = len2 > 0.0 ? 1.0 / sqrt(len2) : 0.0;  // equal pivots: no direction, a slab of 0
    double along = 0.0, abs_sum = 0.0;
    for (int f = 0; f < d; ++f) {
        const double t = (double)piv[hi * dp + f] - (double)piv[lo * dp + f];
        const float u = (float)(t * inv);
        dirs[((int64_t)b * d + f) * K + a] = a > b ? u : -u;  // from b towards a
        along = fma(t, (double)u, along);
        abs_sum += fabs(t * (double)u);
    }
    apart[a * K + b] = __double2float_rd(along - 1e-12 * abs_sum);
}

// Nearest pivot of every point (pivots in shared memory).
template <int DP>
__global__ void __launch_bounds__(kThreads) assign_kernel(const float *__restrict__ xs, int64_t n,
                                                          const float *__restrict__ piv, int K, uint8_t *__restrict__ of) {
    extern __shared__ __align__(16) float smp[];
    float *pn = smp + K * DP;
    for (int e = threadIdx.x; e < K * DP; e += kThreads) smp[e] = -2.f * piv[e];
    __syncthreads();
    for (int k = threadIdx.x; k < K; k += kThreads) {
        float s = 0.f;
        for (int f = 0; f < DP; ++f) s = fmaf(smp[k * DP + f], smp[k * DP + f], s);
        pn[k] = 0.25f * s;
    }
    __syncthreads();
    for (int64_t i = blockIdx.x * (int64_t)kThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kThreads) {
        float4 x[DP / 4];
#pragma unroll
        for (int v = 0; v < DP / 4; ++v) x[v] = reinterpret_cast<const float4 *>(xs + i * DP)[v];
        of[i] = (uint8_t)nearest<DP>(x, reinterpret_cast<const float4 *>(smp), pn, K);
    }
}

// One warp per set; lane l holds the directions of the pivots l, l + 32, ... and goes through the set's points,
// whose offsets from the home pivot it reads as broadcasts.
template <int DP>
__global__ void __launch_bounds__(kThreads) reach_kernel(Cells c, const float *__restrict__ xs, int d, int64_t n,
                                                         const int32_t *__restrict__ order,
                                                         const int32_t *__restrict__ off,
                                                         const int64_t *__restrict__ n_sets_dev, int64_t max_sets,
                                                         int transposed, int32_t *__restrict__ home,
                                                         float *__restrict__ reach) {
    __shared__ __align__(16) float st[kThreads / 32][32][DP];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t n_sets = n_sets_dev ? min(*n_sets_dev, max_sets) : max_sets;
    const int64_t nw = (int64_t)gridDim.x * (kThreads / 32);
    const int K = c.K;
    for (int64_t s = blockIdx.x * (int64_t)(kThreads / 32) + warp; s < n_sets; s += nw) {
        const int64_t r0 = off ? off[s] : s * 128, r1 = off ? off[s + 1] : min((s + 1) * (int64_t)128, n);
        const int b = c.of[order[r0]];
        float r2 = 0.f;
        // up to two passes over the pivots, two directions per lane each
        for (int k0 = 0; k0 < K; k0 += 64) {
            const int a0 = k0 + lane, a1 = a0 + 32;
            float u0[DP], u1[DP];
#pragma unroll
            for (int f = 0; f < DP; ++f) {
                u0[f] = f < d && a0 < K ? c.dirs[((int64_t)b * d + f) * K + a0] : 0.f;
                u1[f] = f < d && a1 < K ? c.dirs[((int64_t)b * d + f) * K + a1] : 0.f;
            }
            float m0 = neg_inf<float>(), m1 = neg_inf<float>();
            for (int64_t r = r0; r < r1; r += 32) {
                const int cnt = (int)min((int64_t)32, r1 - r);
                __syncwarp();
                if (lane < cnt) {
                    const float *x = xs + (int64_t)order[r + lane] * DP;
                    float q = 0.f;
#pragma unroll
                    for (int f = 0; f < DP; ++f) {
                        const float t = x[f] - c.pivots[b * DP + f];
                        st[warp][lane][f] = t;
                        q = fmaf(t, t, q);
                    }
                    r2 = fmaxf(r2, q);
                }
                __syncwarp();
                for (int i = 0; i < cnt; ++i) {
                    float s0 = 0.f, s1 = 0.f;
#pragma unroll
                    for (int f = 0; f < DP; f += 4) {
                        const float4 t = *reinterpret_cast<const float4 *>(&st[warp][i][f]);
                        s0 = fmaf(t.x, u0[f], s0);
                        s1 = fmaf(t.x, u1[f], s1);
                        s0 = fmaf(t.y, u0[f + 1], s0);
                        s1 = fmaf(t.y, u1[f + 1], s1);
                        s0 = fmaf(t.z, u0[f + 2], s0);
                        s1 = fmaf(t.z, u1[f + 2], s1);
                        s0 = fmaf(t.w, u0[f + 3], s0);
                        s1 = fmaf(t.w, u1[f + 3], s1);
                    }
                    m0 = fmaxf(m0, s0);  // NaN coordinates are skipped
                    m1 = fmaxf(m1, s1);
                }
            }
            float rr = r2;
            for (int o = 16; o > 0; o >>= 1) rr = fmaxf(rr, __shfl_xor_sync(0xFFFFFFFFu, rr, o));
            const float err = (float)(d + 8) * 1.1920928955078125e-07f * sqrtf(rr);
            if (a0 < K) reach[transposed ? (int64_t)a0 * max_sets + s : s * K + a0] = __fadd_ru(m0, err);
            if (a1 < K) reach[transposed ? (int64_t)a1 * max_sets + s : s * K + a1] = __fadd_ru(m1, err);
        }
        if (lane == 0) home[s] = b;
    }
}

int grid_of(int64_t threads) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((threads + kThreads - 1) / kThreads, (int64_t)kNumSMsB200 * 8));
}

struct Layout {
    size_t of, piv[2], sum, dirs, apart, total;
};
Layout layout(int64_t n, int d, int K) {
    const int dp = (d + 3) / 4 * 4;
    Layout L{};
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off = align_up(off + bytes, 256);
        return o;
    };
    L.of = take((size_t)n);
    L.piv[0] = take((size_t)K * dp * 4);
    L.piv[1] = take((size_t)K * dp * 4);
    L.sum = take((size_t)kIters * K * (dp + 1) * 4);
    L.dirs = take((size_t)K * K * d * 4);
    L.apart = take((size_t)K * K * 4);
    L.total = off + 256;
    return L;
}

// k-means, directions and the assignment
template <int DP>
cudaError_t launch_build(const float *xs, int64_t n, int d, int K, float *const (&piv)[2], float *sum, float *dirs,
                         float *apart, uint8_t *of, cudaStream_t stream) {
    const int64_t S = sample_size(n);
    const size_t smem = (size_t)(K * DP + K + K * (DP + 1)) * 4;
    for (int it = 0; it <= kIters; ++it) {
        const bool last = it == kIters;
        kmeans_kernel<DP><<<last ? 1 : (unsigned)((S + kMeansThreads - 1) / kMeansThreads), kMeansThreads, smem, stream>>>(
            xs, n, d, K, S, it, piv[(it + 1) & 1], sum + (size_t)std::max(it - 1, 0) * K * (DP + 1), piv[it & 1],
            sum + (size_t)std::min(it, kIters - 1) * K * (DP + 1), last ? 1 : 0);
    }
    directions_kernel<<<K, kMaxCells, 0, stream>>>(piv[kIters & 1], d, DP, K, dirs, apart);
    assign_kernel<DP><<<grid_of(n), kThreads, (size_t)K * (DP + 1) * 4, stream>>>(xs, n, piv[kIters & 1], K, of);
    return cudaGetLastError();
}
template <int DP>
cudaError_t launch_reach(const Cells &c, const float *xs, int d, int64_t n, const int32_t *order, const int32_t *off,
                         const int64_t *n_sets, int64_t max_sets, bool transposed, int32_t *home, float *out,
                         cudaStream_t stream) {
    reach_kernel<DP><<<grid_of(max_sets * 32), kThreads, 0, stream>>>(c, xs, d, n, order, off, n_sets, max_sets,
                                                                     transposed ? 1 : 0, home, out);
    return cudaGetLastError();
}

}  // namespace

int count(int64_t n, int d) {
    if (d < kMinDim || n < kMinPoints) return 0;
    int K = 32;
    while (K < kMaxCells && (int64_t)K * 2 * 4096 <= n) K *= 2;
    return K;
}

size_t workspace(int64_t n, int d) {
    const int K = count(n, d);
    return K == 0 ? 0 : layout(n, d, K).total;
}

nngp_status build(const float *xs, int64_t n, int d, int dp, void *ws, size_t ws_bytes, Cells *out, cudaStream_t stream) {
    const int K = count(n, d);
    if (count(n, d) == 0 || dp != (d + 3) / 4 * 4 || dp > kMaxD)
        return fail(NNGP_ERR_UNSUPPORTED, "knn cells: shape outside the pruned search");
    const Layout L = layout(n, d, K);
    if (!ws || ws_bytes < L.total) return fail(NNGP_ERR_WORKSPACE, "knn cells: workspace too small");
    char *base = reinterpret_cast<char *>(align_up(reinterpret_cast<uintptr_t>(ws), 256));
    float *piv[2] = {reinterpret_cast<float *>(base + L.piv[0]), reinterpret_cast<float *>(base + L.piv[1])};
    float *sum = reinterpret_cast<float *>(base + L.sum);
    NNGP_CUDA_TRY(cudaMemsetAsync(sum, 0, (size_t)kIters * K * (dp + 1) * 4, stream));
    const float *p = piv[kIters & 1];
    float *dirs = reinterpret_cast<float *>(base + L.dirs), *apart = reinterpret_cast<float *>(base + L.apart);
    uint8_t *of = reinterpret_cast<uint8_t *>(base + L.of);
    cudaError_t e = cudaErrorInvalidValue;
    switch (dp) {
        case 12: e = launch_build<12>(xs, n, d, K, piv, sum, dirs, apart, of, stream); break;
        case 16: e = launch_build<16>(xs, n, d, K, piv, sum, dirs, apart, of, stream); break;
        case 20: e = launch_build<20>(xs, n, d, K, piv, sum, dirs, apart, of, stream); break;
        case 24: e = launch_build<24>(xs, n, d, K, piv, sum, dirs, apart, of, stream); break;
    }
    NNGP_CUDA_TRY(e);
    out->K = K;
    out->of = of;
    out->pivots = p;
    out->dirs = dirs;
    out->apart = apart;
    return NNGP_OK;
}

nngp_status reach(const Cells &c, const float *xs, int d, int dp, int64_t n, const int32_t *order, const int32_t *off,
                  const int64_t *n_sets, int64_t max_sets, bool transposed, int32_t *home, float *out,
                  cudaStream_t stream) {
    cudaError_t e = cudaErrorInvalidValue;
    switch (dp) {
        case 12: e = launch_reach<12>(c, xs, d, n, order, off, n_sets, max_sets, transposed, home, out, stream); break;
        case 16: e = launch_reach<16>(c, xs, d, n, order, off, n_sets, max_sets, transposed, home, out, stream); break;
        case 20: e = launch_reach<20>(c, xs, d, n, order, off, n_sets, max_sets, transposed, home, out, stream); break;
        case 24: e = launch_reach<24>(c, xs, d, n, order, off, n_sets, max_sets, transposed, home, out, stream); break;
    }
    NNGP_CUDA_TRY(e);
    return NNGP_OK;
}

}  // namespace cells
}  // namespace nngp
