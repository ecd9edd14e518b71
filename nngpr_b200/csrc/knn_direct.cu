// Direct k-nearest-neighbour search: the refs of a query spread over the threads of a CTA.
//
// Same contract as the other searches (knn.cu): ascending exact distance ((t0^2 + t1^2) + ..., every
// step rounded), lower index first on ties, -1 padding, ref cut; a distance that is NaN or +inf is
// never listed (as in the generic and the SIMT kernel).
//
// Measured (one B200, against the kernel that had the shape before): 2,000 points over themselves
// d = 3 394 -> below 39 us (the host's call time), 256 queries of 16,599 refs d = 18 840 -> 67 us, FP64
// 20,000 points over themselves d = 3 11,651 -> 564 us, d = 20 46.6 -> 1.6 ms.  The bound is the
// FP32 (FP64) issue of the distances: about 0.8 ps a pair at d <= 4, 1.4 at 8, 3.0 at 20 in FP32.
// Points on a grid and repeated points (with ref j in thread j mod 256, lists bounded by the minima alone and
// ties bisected over all refs -> now; 1,000 queries, FP32): 256 x 64 grid 763 -> 46 us, 512 x 64 1,482 -> 65,
// 256 x 1,024 12,114 -> 394, half of 100,000 points in 20 places 3,830 -> 198; 16,384 random points 48 -> 52.
//
// What it is for: searches that are short in queries (a prediction of a few hundred points, a small
// model's fit step), where the other kernels give one thread or one TMEM lane to a query and
// leave most of the chip idle, and the FP64 search, which has no screen.  Nothing of size
// n_query x n_ref is stored; the work is the exact distances (3 d operations a pair) plus one
// compare, and every ref is read once per CTA for its Q queries:
//   1. each of the 256 threads takes one ref of every block of 256 and keeps its K = 3 or 4 nearest per query in
//      registers.  Which one turns from block to block (ref_of): with ref j in thread j mod 256, points on a
//      grid whose rows are 256 long, or any period that divides 256, put a whole column of near refs into one
//      thread, and the bound of step 2 reached sixteen grid steps instead of three;
//   2. the m-th smallest of the 256 thread minima bounds the query's m-th distance from above
//      (each minimum is a distinct ref).  One warp per query finds it by bisection on the high 32
//      bits of the distances, to within 2^12 units;
//   3. kept refs within the bound go to a list in shared memory, normally m plus a few.  A list that is long
//      (repeated points) is bounded again by its own m-th entry, in (distance, index) order, which ends the
//      ties: a thread keeps its lowest indices.  A thread whose K-th kept ref lies before the
//      bound may have dropped some that do: its refs are gone through again, spread over its warp;
//   4. each listed ref's rank (entries before it in (distance, index) order) is its place.
// A list that overflows in step 3 (near refs in few threads all the same) is bounded by its m-th entry as well and
// filled again, every time with at least kCap - m refs fewer.
#include <algorithm>

#include "common.cuh"
#include "knn_direct.cuh"

namespace nngp {
namespace direct {
namespace {

constexpr int kThreads = 256;
// Refs that a thread keeps per query.  Some thread has three of a query's 32 near ones in about one query of ten, and
// its refs are gone through again; four in one of 300.  With one query per CTA the fourth is free (256 queries of
// 16,599, d = 18, 56.9 -> 54.5 us; 1,000 of 8,000, d = 8, 35.3 -> 31.9); with four it costs registers and
// shared memory (16,384 points over themselves, d = 3, 197 -> 237 us).
template <int Q> constexpr int kKeep = Q == 1 ? 4 : 3;
template <int Q> constexpr int kCap = kKeep<Q> * kThreads;  // every thread's kept refs
constexpr int kLong = kThreads;         // a longer list is bounded by its own m-th entry first
constexpr uint32_t kTol = 1u << 12;
constexpr uint32_t kNone = 0xFFFFFFFFu;  // no finite distance

// the high 32 bits of a non-negative distance: integer order = distance order
__device__ __forceinline__ uint32_t high_bits(float v) { return __float_as_uint(v); }
__device__ __forceinline__ uint32_t high_bits(double v) { return (uint32_t)__double2hiint(v); }
__device__ __forceinline__ uint64_t all_bits(float v) { return __float_as_uint(v); }
__device__ __forceinline__ uint64_t all_bits(double v) { return (uint64_t)__double_as_longlong(v); }

__device__ __forceinline__ float from_bits(uint64_t b, float) { return __uint_as_float((uint32_t)b); }
__device__ __forceinline__ double from_bits(uint64_t b, double) { return __longlong_as_double((long long)b); }
// the largest distance with these high bits (high_bits); +inf for kNone - 1
__device__ __forceinline__ float up_to(uint32_t h, float) {
    return h < 0x7F800000u ? __uint_as_float(h) : pos_inf<float>();
}
__device__ __forceinline__ double up_to(uint32_t h, double) {
    return h < 0x7FF00000u ? __hiloint2double((int)h, -1) : pos_inf<double>();
}

// Which ref of block k (refs 256 k .. 256 k + 255) a thread has: tid ^ ref_of(k).  The low 8 bits are a hash of k, so
// that refs whose indices differ by a multiple of 256 share a thread for about one pair of blocks in 256.  A thread
// that has G blocks in flight takes one hash for them, 64 refs apart (one query per CTA, 1,000 queries of 434,874
// refs, d = 3: 660 us with a hash for each block, 593 so, 533 without any).
__device__ __forceinline__ uint32_t turn(int g) {
    uint32_t h = (uint32_t)g * 0x9E3779B1u;
    h = (h ^ (h >> 15)) * 0x85EBCA6Bu;
    return h >> 24;
}
template <int G> __device__ __forceinline__ int ref_of(int k) {
    static_assert(G == 1 || G == 4, "blocks in flight");
    return k * kThreads + (int)(turn(k / G) ^ (uint32_t)(k % G * 64));
}

// (distance, index) order
template <typename T> __device__ __forceinline__ bool before(T d, int j, T bd, int bj) {
    return d < bd || (d == bd && j < bj);
}

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

// The m-th smallest of c list entries in (distance, index) order, found by one warp: bisection on the distance's
// bits, then on the index among the entries at that distance.  (+inf, INT32_MAX) when c < m.
template <typename T>
__device__ __forceinline__ void mth_entry(const T *cd, const int32_t *cj, int c, int m, int lane, T &bd, int &bj) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    bd = pos_inf<T>();
    bj = INT32_MAX;
    if (c < m) return;
    auto count = [&](auto &&in) -> int {
        unsigned n = 0;
        for (int e = lane; e < c; e += 32) n += in(cd[e], cj[e]) ? 1u : 0u;
        return (int)__reduce_add_sync(FULL, n);
    };
    T mn = pos_inf<T>(), mx = T(0);
    for (int e = lane; e < c; e += 32) {
        mn = cd[e] < mn ? cd[e] : mn;
        mx = cd[e] > mx ? cd[e] : mx;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const T a = __shfl_xor_sync(FULL, mn, o), b = __shfl_xor_sync(FULL, mx, o);
        mn = a < mn ? a : mn;
        mx = b > mx ? b : mx;
    }
    uint64_t lo = all_bits(mn), hi = all_bits(mx);
    while (lo < hi) {
        const uint64_t mid = lo + ((hi - lo) >> 1);
        const T v = from_bits(mid, T());
        if (count([&](T d, int) { return d <= v; }) >= m) hi = mid;
        else lo = mid + 1;
    }
    bd = from_bits(lo, T());
    const T v = bd;
    const int left = m - count([&](T d, int) { return d < v; });  // of the entries at that distance
    int jl = 0, jh = INT32_MAX;
    while (jl < jh) {
        const int mid = jl + ((jh - jl) >> 1);
        if (count([&](T d, int j) { return d == v && j <= mid; }) >= left) jh = mid;
        else jl = mid + 1;
    }
    bj = jl;
}

// What the threads of a CTA share: its Q queries and, of each, a list of refs and the list's bound, up to (bd, bj).
// DP: row length when it is known at compile time (0: any).
template <typename T, int DP, int Q> struct Shared {
    alignas(32) T q[Q][DP > 0 ? DP : 256];
    alignas(16) T d[Q][kCap<Q>];
    int32_t j[Q][kCap<Q>];
    int count[Q];  // refs pushed; the first kCap of them are listed
    T bd[Q];
    int bj[Q];
    unsigned more;  // queries whose list is not final

    __device__ __forceinline__ bool within(int i, T dist, int ref) const { return !before(bd[i], bj[i], dist, ref); }
    __device__ __forceinline__ void push(int i, T dist, int ref) {
        const int at = atomicAdd(&count[i], 1);
        if (at < kCap<Q>) {
            d[i][at] = dist;
            j[i][at] = ref;
        }
    }
};
// A thread's nearest refs of a query, in (distance, index) order; j < 0: none.
template <typename T, int K> struct Kept {
    T d[K];
    int j[K];
    // may the thread have dropped refs that lie before (bd, bj)?
    __device__ __forceinline__ bool dropped(T bd, int bj) const {
        return j[K - 1] >= 0 && before(d[K - 1], j[K - 1], bd, bj);
    }
};

// Step 3 for the lists that are long, or whose threads may have dropped refs (todo: a bit per query, the same in
// every thread): a call of its own, so that it holds no register of the distance loop.
template <int G, typename T, int DP, int Q>
__device__ __noinline__ void refine(Shared<T, DP, Q> &sh, const Kept<T, kKeep<Q>> *kept, const int *lim, unsigned todo,
                                    const T *__restrict__ refs, int n_ref, int blocks, int dp_any, int m) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    constexpr int R = 2;  // refs of a lane in flight
    constexpr int K = kKeep<Q>;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int dp = DP > 0 ? DP : dp_any;
    while (todo) {
        unsigned again = 0;  // lists that are bounded by their own m-th entry and start anew
        for (int q = 0; q < Q; ++q) again |= ((todo >> q) & 1u) && sh.count[q] > kLong ? 1u << q : 0u;
        __syncthreads();  // every thread has read the counts
        if (again) {
            if (warp < Q && ((again >> warp) & 1u)) {
                T bd;
                int bj;
                mth_entry(sh.d[warp], sh.j[warp], min(sh.count[warp], kCap<Q>), m, lane, bd, bj);
                __syncwarp();
                if (lane == 0) {
                    sh.bd[warp] = bd;
                    sh.bj[warp] = bj;
                    sh.count[warp] = 0;
                }
            }
            __syncthreads();
            for (int q = 0; q < Q; ++q)
                for (int k = 0; ((again >> q) & 1u) && k < K; ++k) {
                    const T d = kept[q].d[k];
                    const int j = kept[q].j[k];
                    if (j >= 0 && sh.within(q, d, j)) sh.push(q, d, j);
                }
        }
        unsigned scan = 0;  // queries for which this thread's refs are gone through again
        for (int q = 0; q < Q; ++q)
            if (((todo >> q) & 1u) && kept[q].dropped(sh.bd[q], sh.bj[q])) scan |= 1u << q;
        // the refs of one such thread after the other, spread over its warp
        for (unsigned left = __ballot_sync(FULL, scan != 0); left; left &= left - 1) {
            const int src = __ffs((int)left) - 1;
            const unsigned qs = __shfl_sync(FULL, scan, src);
            T ld[Q];  // the last kept ref: those up to it are listed
            int lj[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                ld[q] = __shfl_sync(FULL, kept[q].d[K - 1], src);
                lj[q] = __shfl_sync(FULL, kept[q].j[K - 1], src);
            }
            for (int k0 = lane; k0 < blocks; k0 += 32 * R) {
                int jr[R];
                const T *row[R];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    jr[r] = (warp * 32 + src) ^ ref_of<G>(k0 + 32 * r);
                    row[r] = refs + (int64_t)min(jr[r], n_ref - 1) * dp;
                }
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    if (!((qs >> q) & 1u)) continue;
                    T s[R];
#pragma unroll
                    for (int f = 0; f < dp; f += 4) {
                        const Vec4<T> u = load4(&sh.q[q][f]);
#pragma unroll
                        for (int r = 0; r < R; ++r) s[r] = add4(s[r], load4(row[r] + f), u, f == 0);
                    }
#pragma unroll
                    for (int r = 0; r < R; ++r)
                        if (s[r] < pos_inf<T>() && jr[r] < lim[q] && before(ld[q], lj[q], s[r], jr[r]) &&
                            sh.within(q, s[r], jr[r]))
                            sh.push(q, s[r], jr[r]);
                }
            }
        }
        __syncthreads();
        for (int q = 0; q < Q; ++q)
            if (((todo >> q) & 1u) && sh.count[q] <= kCap<Q>) todo &= ~(1u << q);
    }
}

// CTAs per SM that the registers are held to (0: no limit), where the compiler's own choice was slower: 16,384 points
// over themselves, d = 3, 214 -> 204 us; 20,000, d = 40, 2,192 -> 1,474 us.
template <typename T, int DP, int Q>
constexpr int kMinCtas = Q == 4 && sizeof(T) == 4 ? (DP == 4 ? 5 : (DP == 0 ? 3 : 0)) : 0;

// Q queries per CTA, R refs per thread in flight (Q * R independent sums hide the latency of the serial additions).
template <typename T, int DP, int Q, int R>
__global__ void __launch_bounds__(kThreads, (kMinCtas<T, DP, Q>))
    knn_direct_kernel(const T *__restrict__ refs, const T *__restrict__ qs, int64_t n_query, int64_t n_ref, int dp_any,
                      int has_cut, int64_t cut, int m, int32_t *__restrict__ out) {
    constexpr int K = kKeep<Q>;
    __shared__ Shared<T, DP, Q> sh;
    uint32_t(*smin)[kThreads] = reinterpret_cast<uint32_t(*)[kThreads]>(&sh.d[0][0]);  // in the lists' place
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
        sh.q[q][e - q * dp] = q < nq ? qs[(q0 + q) * dp + (e - q * dp)] : T(0);
    }
    if (tid < Q) sh.count[tid] = 0;
    if (tid == 0) sh.more = 0;
    int lim[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) lim[q] = q < nq ? limit_of(q0 + q) : 0;
    const int lim_max = limit_of(q0 + nq - 1);  // limits ascend
    __syncthreads();

    Kept<T, K> kept[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
        for (int k = 0; k < K; ++k) {
            kept[q].d[k] = pos_inf<T>();
            kept[q].j[k] = -1;
        }
    const int blocks = (int)(((int64_t)lim_max + kThreads - 1) / kThreads);
    for (int k0 = 0; k0 < blocks; k0 += R) {
        const uint32_t h = turn(k0 / R);
        T s[Q][R];
        int jr[R];
        const T *row[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            jr[r] = tid ^ ((k0 + r) * kThreads + (int)(h ^ (uint32_t)(r * 64)));  // ref_of<R>(k0 + r)
            row[r] = refs + (int64_t)min(jr[r], (int)n_ref - 1) * dp;
        }
        auto group = [&](int f) {
            Vec4<T> v[R];
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = load4(row[r] + f);
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const Vec4<T> u = load4(&sh.q[q][f]);
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
                const int j = jr[r];
                const T d = s[q][r];
                if (d < kept[q].d[K - 1] && j < lim[q]) {  // NaN and +inf never; ties keep the lower index
                    Kept<T, K> &kp = kept[q];
                    if constexpr (K == 3) {  // spelled out: the loops below cost the four-query form 1 to 5 %
                        const bool b0 = d < kp.d[0], b1 = d < kp.d[1];
                        kp.d[2] = b1 ? kp.d[1] : d;
                        kp.j[2] = b1 ? kp.j[1] : j;
                        kp.d[1] = b0 ? kp.d[0] : (b1 ? d : kp.d[1]);
                        kp.j[1] = b0 ? kp.j[0] : (b1 ? j : kp.j[1]);
                        kp.d[0] = b0 ? d : kp.d[0];
                        kp.j[0] = b0 ? j : kp.j[0];
                    } else {
                        bool b[K];  // d lies before the k-th kept
#pragma unroll
                        for (int k = 0; k < K; ++k) b[k] = k == K - 1 || d < kp.d[k];
#pragma unroll
                        for (int k = K - 1; k > 0; --k) {
                            kp.d[k] = b[k - 1] ? kp.d[k - 1] : (b[k] ? d : kp.d[k]);
                            kp.j[k] = b[k - 1] ? kp.j[k - 1] : (b[k] ? j : kp.j[k]);
                        }
                        kp.d[0] = b[0] ? d : kp.d[0];
                        kp.j[0] = b[0] ? j : kp.j[0];
                    }
                }
            }
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) smin[q][tid] = kept[q].j[0] >= 0 ? high_bits(kept[q].d[0]) : kNone;
    __syncthreads();
    if (warp < Q) {
        const uint32_t b = mth_of_256(smin[warp], m, lane);
        if (lane == 0) {
            sh.bd[warp] = up_to(b, T());
            sh.bj[warp] = INT32_MAX;
        }
    }
    __syncthreads();
    unsigned more = 0;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const T bd = sh.bd[q];
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (kept[q].j[k] >= 0 && kept[q].d[k] <= bd) sh.push(q, kept[q].d[k], kept[q].j[k]);
        if (kept[q].dropped(bd, INT32_MAX)) more |= 1u << q;
    }
    if (more) atomicOr(&sh.more, more);
    __syncthreads();
    unsigned todo = sh.more;
#pragma unroll
    for (int q = 0; q < Q; ++q) todo |= sh.count[q] > kLong ? 1u << q : 0u;
    if (todo) {
        Kept<T, K> mine[Q];  // copies, so that only these are in memory
        int lims[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            mine[q] = kept[q];
            lims[q] = lim[q];
        }
        refine<R>(sh, mine, lims, todo, refs, (int)n_ref, blocks, dp, m);
    }
    for (int q = 0; q < nq; ++q) {
        const int c = sh.count[q];
        int32_t *o = out + (q0 + q) * m;
        for (int e = tid; e < c; e += kThreads) {
            const T d = sh.d[q][e];
            const int j = sh.j[q][e];
            int rank = 0;
            for (int k = 0; k < c; ++k) {
                const T dk = sh.d[q][k];
                rank += (dk < d || (dk == d && sh.j[q][k] < j)) ? 1 : 0;
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
        knn_direct_kernel<T, DP, 1, 4><<<(unsigned)n_query, kThreads, 0, stream>>>(refs, qs, n_query, n_ref, dp,
                                                                                 has_cut, cut, m, out);
    return cudaGetLastError();
}

}  // namespace

template <typename T>
nngp_status search(const T *refs, int64_t n_ref, const T *qs, int64_t n_query, int d, int m, int has_cut, int64_t cut,
                   int32_t *out, cudaStream_t stream) {
    static_assert(kMaxNeighbours <= kLong && kMaxNeighbours <= kThreads, "the bound needs m thread minima");
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
