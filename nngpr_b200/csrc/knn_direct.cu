// Direct k-nearest-neighbour search: the refs of a query spread over the threads of a CTA.
//
// Same contract as the other searches (knn.cu): ascending exact distance ((t0^2 + t1^2) + ..., every
// step rounded), lower index first on ties, -1 padding, ref cut; a distance that is NaN or +inf is
// never listed (as in the generic and the SIMT kernel).
//
// Measured (one B200, against the kernel that had the shape before): 2,000 points over themselves
// d = 3 394 -> below 39 us (the host's call time), 256 queries of 16,599 refs d = 18 840 -> 67 us, FP64
// 20,000 points over themselves d = 3 11,651 -> 586 us, d = 20 46.6 -> 1.7 ms.  The bound is the
// FP32 (FP64) issue of the distances: about 0.8 ps a pair at d <= 4, 1.4 at 8, 3.0 at 20 in FP32.
//
// What it is for: searches that are short in queries (a prediction of a few hundred points, a small
// model's fit step), where the other kernels give one thread or one TMEM lane to a query and
// leave most of the chip idle, and the FP64 search, which has no screen.  Nothing of size
// n_query x n_ref is stored; the work is the exact distances (3 d operations a pair) plus one
// compare, and every ref is read once per CTA for its Q queries:
//   1. each of the 256 threads takes the refs j = tid, tid + 256, ... and keeps its K = 3 nearest per
//      query in registers;
//   2. the m-th smallest of the 256 thread minima bounds the query's m-th distance from above
//      (each minimum is a distinct ref).  One warp per query finds it by bisection on the high 32
//      bits of the distances, to within 2^12 units;
//   3. kept refs within the bound go to a list in shared memory, normally m plus a few: the refs
//      of a query's list are rarely in the same thread (consecutive indices are in consecutive
//      threads).  A thread whose K-th kept ref is still within the bound may have dropped some and
//      goes through its refs again;
//   4. each listed ref's rank (entries before it in (distance, index) order) is its place.
// More than kCap refs within the bound (exact ties: lattices, duplicates) take a bisection on the
// whole distance, then on the index of the refs at the m-th distance, over recomputed
// distances: as exact, slower.
#include <algorithm>

#include "common.cuh"
#include "knn_direct.cuh"

namespace nngp {
namespace direct {
namespace {

constexpr int kThreads = 256;
constexpr int kKeep = 3;
constexpr int kCap = 512;
constexpr uint32_t kTol = 1u << 12;
constexpr uint32_t kNone = 0xFFFFFFFFu;  // no finite distance

// the high 32 bits of a non-negative distance: integer order = distance order
__device__ __forceinline__ uint32_t high_bits(float v) { return __float_as_uint(v); }
__device__ __forceinline__ uint32_t high_bits(double v) { return (uint32_t)__double2hiint(v); }
__device__ __forceinline__ uint64_t all_bits(float v) { return __float_as_uint(v); }
__device__ __forceinline__ uint64_t all_bits(double v) { return (uint64_t)__double_as_longlong(v); }

template <typename T> struct Vec4 {
    T x, y, z, w;
};
__device__ __forceinline__ Vec4<float> load4(const float *p) {
    const float4 v = *reinterpret_cast<const float4 *>(p);
    return {v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ Vec4<double> load4(const double *p) {
    const double2 a = reinterpret_cast<const double2 *>(p)[0], b = reinterpret_cast<const double2 *>(p)[1];
    return {a.x, a.y, b.x, b.y};
}

// adds four features to the running sum (the first group starts it); features past d are zero in
// both rows and add exact zeros
template <typename T>
__device__ __forceinline__ T add4(T s, const Vec4<T> &r, const Vec4<T> &q, bool first) {
    T t = sub_rn(r.x, q.x);
    s = first ? mul_rn(t, t) : add_rn(s, mul_rn(t, t));
    t = sub_rn(r.y, q.y);
    s = add_rn(s, mul_rn(t, t));
    t = sub_rn(r.z, q.z);
    s = add_rn(s, mul_rn(t, t));
    t = sub_rn(r.w, q.w);
    return add_rn(s, mul_rn(t, t));
}

// The m-th smallest of 256 values (8 per lane of one warp; kNone never counts), or an upper bound of it
// within kTol; kNone - 1 when fewer than m values count.
__device__ __forceinline__ uint32_t mth_of_256(const uint32_t *v256, int m, int lane) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    uint32_t v[kThreads / 32];
    uint32_t mn = kNone, mx = 0u;
#pragma unroll
    for (int e = 0; e < kThreads / 32; ++e) {
        v[e] = v256[e * 32 + lane];
        if (v[e] != kNone) {
            mn = min(mn, v[e]);
            mx = max(mx, v[e]);
        }
    }
    auto count_le = [&](uint32_t bound) -> int {
        unsigned c = 0;
#pragma unroll
        for (int e = 0; e < kThreads / 32; ++e) c += v[e] <= bound ? 1u : 0u;
        return (int)__reduce_add_sync(FULL, c);
    };
    if (count_le(kNone - 1) < m) return kNone - 1;
    uint32_t lo = __reduce_min_sync(FULL, mn), hi = __reduce_max_sync(FULL, mx);
    while (hi - lo > kTol) {  // count_le(hi) >= m throughout
        const uint32_t mid = lo + ((hi - lo) >> 1);
        if (count_le(mid) >= m) hi = mid;
        else lo = mid + 1;
    }
    return hi;
}

// DP: row length when it is known at compile time (0: any); Q queries per CTA, R refs per thread in flight
// (Q * R independent sums hide the latency of the serial additions).
template <typename T, int DP, int Q, int R>
__global__ void __launch_bounds__(kThreads) knn_direct_kernel(const T *__restrict__ refs, const T *__restrict__ qs,
                                                              int64_t n_query, int64_t n_ref, int dp_any, int has_cut,
                                                              int64_t cut, int m, int32_t *__restrict__ out) {
    constexpr int QROW = DP > 0 ? DP : 256;
    __shared__ __align__(32) T sq[Q][QROW];
    __shared__ uint32_t smin[Q][kThreads];
    __shared__ uint32_t sbound[Q];
    __shared__ int scount[Q];
    __shared__ T cd[Q][kCap];
    __shared__ int32_t cj[Q][kCap];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int dp = DP > 0 ? DP : dp_any;
    // prefix searches: the queries with the most refs first
    const int64_t blk = has_cut ? (int64_t)(gridDim.x - 1 - blockIdx.x) : (int64_t)blockIdx.x;
    const int64_t q0 = blk * Q;
    const int nq = (int)min((int64_t)Q, n_query - q0);
    auto limit_of = [&](int64_t q) -> int {
        if (!has_cut) return (int)n_ref;
        const int64_t l = q + cut;
        return (int)(l < 0 ? 0 : (l > n_ref ? n_ref : l));
    };
    for (int e = tid; e < Q * dp; e += kThreads) {
        const int q = e / dp;
        sq[q][e - q * dp] = q < nq ? qs[(q0 + q) * dp + (e - q * dp)] : T(0);
    }
    if (tid < Q) scount[tid] = 0;
    int lim[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) lim[q] = q < nq ? limit_of(q0 + q) : 0;
    const int lim_max = limit_of(q0 + nq - 1);  // limits ascend
    __syncthreads();

    // distance of ref j to query q (rescans)
    auto dist = [&](int q, int j) -> T {
        const T *row = refs + (int64_t)j * dp;
        T s = T(0);
        for (int f = 0; f < dp; f += 4) s = add4(s, load4(row + f), load4(&sq[q][f]), f == 0);
        return s;
    };

    T kd[Q][kKeep];
    int kj[Q][kKeep];
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
        for (int k = 0; k < kKeep; ++k) {
            kd[q][k] = pos_inf<T>();
            kj[q][k] = -1;
        }
    for (int j0 = tid; j0 < lim_max; j0 += kThreads * R) {
        T s[Q][R];
        const T *row[R];
#pragma unroll
        for (int r = 0; r < R; ++r) row[r] = refs + (int64_t)min(j0 + r * kThreads, (int)n_ref - 1) * dp;
        auto group = [&](int f) {
            Vec4<T> v[R];
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = load4(row[r] + f);
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const Vec4<T> u = load4(&sq[q][f]);
#pragma unroll
                for (int r = 0; r < R; ++r) s[q][r] = add4(s[q][r], v[r], u, f == 0);
            }
        };
        if constexpr (DP > 0) {
#pragma unroll
            for (int f = 0; f < DP; f += 4) group(f);
        } else {
            for (int f = 0; f < dp; f += 4) group(f);
        }
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int j = j0 + r * kThreads;
                const T d = s[q][r];
                if (d < kd[q][kKeep - 1] && j < lim[q]) {  // NaN and +inf never; ties keep the lower index
                    const bool b0 = d < kd[q][0], b1 = d < kd[q][1];
                    kd[q][2] = b1 ? kd[q][1] : d;
                    kj[q][2] = b1 ? kj[q][1] : j;
                    kd[q][1] = b0 ? kd[q][0] : (b1 ? d : kd[q][1]);
                    kj[q][1] = b0 ? kj[q][0] : (b1 ? j : kj[q][1]);
                    kd[q][0] = b0 ? d : kd[q][0];
                    kj[q][0] = b0 ? j : kj[q][0];
                }
            }
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) smin[q][tid] = kj[q][0] >= 0 ? high_bits(kd[q][0]) : kNone;
    __syncthreads();
    if (warp < Q) {
        const uint32_t b = mth_of_256(smin[warp], m, lane);
        if (lane == 0) sbound[warp] = b;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const uint32_t bound = sbound[q];
        auto push = [&](T d, int j) {
            const int at = atomicAdd(&scount[q], 1);
            if (at < kCap) {
                cd[q][at] = d;
                cj[q][at] = j;
            }
        };
        if (kj[q][kKeep - 1] >= 0 && high_bits(kd[q][kKeep - 1]) <= bound) {
            for (int j = tid; j < lim[q]; j += kThreads) {
                const T d = dist(q, j);
                if (d < pos_inf<T>() && high_bits(d) <= bound) push(d, j);
            }
        } else {
#pragma unroll
            for (int k = 0; k < kKeep; ++k)
                if (kj[q][k] >= 0 && high_bits(kd[q][k]) <= bound) push(kd[q][k], kj[q][k]);
        }
    }
    __syncthreads();
    for (int q = 0; q < nq; ++q) {
        int c = scount[q];
        if (c > kCap) {  // ties: CTA-uniform
            const int limit = limit_of(q0 + q);
            // refs with distance bits < v, or (at v) index <= jmax; v and jmax the same in every thread
            auto count = [&](uint64_t v, int jmax) -> int {
                int n = 0;
                for (int j = tid; j < limit; j += kThreads) {
                    const T d = dist(q, j);
                    if (d < pos_inf<T>()) {
                        const uint64_t b = all_bits(d);
                        n += (b < v || (b == v && j <= jmax)) ? 1 : 0;
                    }
                }
                __syncthreads();
                if (tid == 0) scount[q] = 0;
                __syncthreads();
                n = (int)__reduce_add_sync(0xFFFFFFFFu, (unsigned)n);
                if (lane == 0 && n > 0) atomicAdd(&scount[q], n);
                __syncthreads();
                return scount[q];
            };
            uint64_t lo = 0, hi = all_bits(pos_inf<T>());  // more than kCap >= m refs are finite
            while (lo < hi) {
                const uint64_t mid = lo + ((hi - lo) >> 1);
                if (count(mid, INT32_MAX) >= m) hi = mid;
                else lo = mid + 1;
            }
            const uint64_t v = lo;
            int jl = 0, jh = limit - 1;
            while (jl < jh) {
                const int mid = jl + ((jh - jl) >> 1);
                if (count(v, mid) >= m) jh = mid;
                else jl = mid + 1;
            }
            __syncthreads();
            if (tid == 0) scount[q] = 0;
            __syncthreads();
            for (int j = tid; j < limit; j += kThreads) {
                const T d = dist(q, j);
                if (!(d < pos_inf<T>())) continue;
                const uint64_t b = all_bits(d);
                if (b < v || (b == v && j <= jl)) {
                    const int at = atomicAdd(&scount[q], 1);
                    cd[q][at] = d;  // exactly m <= kMaxNeighbours <= kCap entries
                    cj[q][at] = j;
                }
            }
            __syncthreads();
            c = scount[q];
        }
        int32_t *o = out + (q0 + q) * m;
        for (int e = tid; e < c; e += kThreads) {
            const T d = cd[q][e];
            const int j = cj[q][e];
            int rank = 0;
            for (int k = 0; k < c; ++k) {
                const T dk = cd[q][k];
                rank += (dk < d || (dk == d && cj[q][k] < j)) ? 1 : 0;
            }
            if (rank < m) o[rank] = j;
        }
        for (int k = c + tid; k < m; k += kThreads) o[k] = -1;
    }
}

template <typename T, int DP>
cudaError_t launch(const T *refs, int64_t n_ref, const T *qs, int64_t n_query, int dp, int m, int has_cut, int64_t cut,
                   int32_t *out, cudaStream_t stream) {
    // four queries share each ref that is read once there are CTAs for every SM that way
    if (n_query >= 4 * 2 * kNumSMsB200)
        knn_direct_kernel<T, DP, 4, 1><<<(unsigned)((n_query + 3) / 4), kThreads, 0, stream>>>(
            refs, qs, n_query, n_ref, dp, has_cut, cut, m, out);
    else
        knn_direct_kernel<T, DP, 1, 4><<<(unsigned)n_query, kThreads, 0, stream>>>(refs, qs, n_query, n_ref, dp, has_cut,
                                                                                 cut, m, out);
    return cudaGetLastError();
}

}  // namespace

template <typename T>
nngp_status search(const T *refs, int64_t n_ref, const T *qs, int64_t n_query, int d, int m, int has_cut, int64_t cut,
                   int32_t *out, cudaStream_t stream) {
    static_assert(kMaxNeighbours <= kCap && kMaxNeighbours <= kThreads, "the bound needs m thread minima");
    if (m < 1 || m > kMaxNeighbours || n_ref < 1 || n_query < 1)
        return fail(NNGP_ERR_UNSUPPORTED, "knn: shape outside the direct search");
    const int dp = row_len(d);
    cudaError_t e = cudaSuccess;
    switch (dp) {
#define NNGP_DIRECT(DD) \
    case DD: e = launch<T, DD>(refs, n_ref, qs, n_query, dp, m, has_cut, cut, out, stream); break;
        NNGP_DIRECT(4) NNGP_DIRECT(8) NNGP_DIRECT(12) NNGP_DIRECT(16) NNGP_DIRECT(20) NNGP_DIRECT(24) NNGP_DIRECT(32)
#undef NNGP_DIRECT
        default: e = launch<T, 0>(refs, n_ref, qs, n_query, dp, m, has_cut, cut, out, stream);
    }
    NNGP_CUDA_TRY(e);
    return NNGP_OK;
}

template nngp_status search<float>(const float *, int64_t, const float *, int64_t, int, int, int, int64_t, int32_t *,
                                   cudaStream_t);
template nngp_status search<double>(const double *, int64_t, const double *, int64_t, int, int, int, int64_t, int32_t *,
                                    cudaStream_t);

}  // namespace direct
}  // namespace nngp
