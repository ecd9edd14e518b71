// Seed thresholds for the prefix neighbour search of the fit step.
//
// The search keeps, for every point i, the m nearest of the points j < i (calc_nn with
// ref_cut_index = 0, nngpr/cuda_kernel_accelerators.py:663-743, as called by
// nngpr/base_nngpr.py:530-535).  The tensor-core kernel streams the refs in index order and
// screens each against the row's current bound, the m-th best distance found so far; in random
// input order a row meets about m ln(i/m) list updates, and every one costs an exact rescoring
// and a list insert.  That candidate work, not the screen, dominates the kernel at small d.
//
// Any m distinct refs j < i bound the row from above: the m-th smallest of their distances is
// >= the m-th smallest over all j < i.  This file finds such refs cheaply: two space-filling
// (Morton) orders of the scaled points, the second on a shifted grid, and for each point the
// refs within W positions of it in either order.  With the m-th smallest of those distances as
// the row's starting bound the screen passes about 40 refs per row instead of about 300 (d = 3,
// uniform data, W = 256).  The bound is computed with exactly the arithmetic of the search's
// exact rescoring, so it never excludes a true neighbour and the lists are bit-identical with or
// without seeds; only the number of candidates changes.
//
// Steps (all on the caller's stream): per-dimension bounds of the finite coordinates; 64-bit
// Morton keys (b = min(10, 64 / d) bits per dimension, interleaved) for both grids; one radix
// sort of both (CUB, key/index pairs); the inverse permutations and the coordinates in either order; then one
// warp per point, points taken in curve order so that neighbouring warps read the same windows.
#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <climits>
#include <cstdlib>
#include <string>

#include "common.cuh"
#include "knn_seed.cuh"

namespace nngp {
namespace seed {
namespace {

constexpr int kThreads = 256;
constexpr uint32_t kInfBits = 0x7F800000u;
constexpr uint32_t kTolBits = 1u << 12;  // stop the bisection within 2^12 ulp (5e-4 relative)

// monotone unsigned image of a float (for atomic min / max) and back
__device__ __forceinline__ uint32_t ord_of(float x) {
    const uint32_t u = __float_as_uint(x);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float from_ord(uint32_t o) {
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7FFFFFFFu) : ~o);
}

// Bounds of the finite coordinates of every feature, as ord_of images.  A thread keeps to one 4-feature column of the
// rows, so that a warp reads whole sectors (a thread per row, feature after feature, took 20.5 against
// 9.4 us at n = 434,874, d = 3, 8.5 against 3.3 at n = 16,599, d = 18).
__global__ void __launch_bounds__(kThreads) bounds_kernel(const float *__restrict__ xs, int64_t n, int d, int dp,
                                                          uint32_t *__restrict__ lo, uint32_t *__restrict__ hi) {
    __shared__ uint32_t slo[256], shi[256];
    slo[threadIdx.x] = 0xFFFFFFFFu;
    shi[threadIdx.x] = 0u;
    __syncthreads();
    const int v4 = dp / 4;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x / v4 * v4;
    const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const float4 *src = reinterpret_cast<const float4 *>(xs);
    if (t0 < stride && t0 < n * v4) {
        uint32_t mn[4] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, mx[4] = {0u, 0u, 0u, 0u};
        auto take = [&](int c, float v) {
            if (isfinite(v)) {
                const uint32_t o = ord_of(v);
                mn[c] = min(mn[c], o);
                mx[c] = max(mx[c], o);
            }
        };
#pragma unroll 4
        for (int64_t t = t0; t < n * v4; t += stride) {
            const float4 r = __ldg(src + t);
            take(0, r.x);
            take(1, r.y);
            take(2, r.z);
            take(3, r.w);
        }
        const int f0 = 4 * (int)(t0 % v4);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (f0 + c < d && mn[c] <= mx[c]) {
                atomicMin(slo + f0 + c, mn[c]);
                atomicMax(shi + f0 + c, mx[c]);
            }
        }
    }
    __syncthreads();
    if ((int)threadIdx.x < d && slo[threadIdx.x] <= shi[threadIdx.x]) {
        atomicMin(lo + threadIdx.x, slo[threadIdx.x]);
        atomicMax(hi + threadIdx.x, shi[threadIdx.x]);
    }
}

// The two grids over the bounds: cells aligned with the bounds (curve 0), and shifted by 1.23 % of the extent in
// every dimension (curve 1).
struct Grids {
    float scale, shift1;
    uint32_t qmax;
};
__device__ __forceinline__ Grids grids_of(const uint32_t *__restrict__ lo, const uint32_t *__restrict__ hi, int d, int bits) {
    float span = 0.f;
    for (int f = 0; f < d; ++f) {
        if (hi[f] >= lo[f]) span = fmaxf(span, from_ord(hi[f]) - from_ord(lo[f]));
    }
    const float cells = (float)(1u << bits);
    return {span > 0.f && isfinite(span) ? 0.97f * cells / span : 0.f, 0.0123f * cells, (1u << bits) - 1u};
}
// A point's Morton key on grid `curve`, without its `drop` lowest bits.
__device__ __forceinline__ uint64_t morton(const float *__restrict__ x, const Grids &g, const uint32_t *__restrict__ lo,
                                           const uint32_t *__restrict__ hi, int d, int bits, int drop, int curve) {
    uint64_t key = 0;
    for (int f = 0; f < d; ++f) {
        const float base = hi[f] >= lo[f] ? from_ord(lo[f]) : 0.f;
        const float t = (x[f] - base) * g.scale + (curve == 0 ? 0.f : g.shift1);
        const uint32_t q = t > 0.f ? (t < (float)g.qmax ? (uint32_t)t : g.qmax) : 0u;  // NaN -> 0
        for (int b = 0; b < bits; ++b) key |= (uint64_t)((q >> b) & 1u) << (b * d + f);
    }
    return key >> drop;
}

// Sort entries of the points on both grids: keys[c n + i] = c above the key of point i on grid c, idx = i.
__global__ void __launch_bounds__(kThreads) keys_kernel(const float *__restrict__ xs, int64_t n, int d, int dp,
                                                        const uint32_t *__restrict__ lo, const uint32_t *__restrict__ hi,
                                                        int bits, int drop, uint64_t *__restrict__ keys,
                                                        int32_t *__restrict__ idx) {
    const Grids g = grids_of(lo, hi, d, bits);
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < 2 * n; e += (int64_t)gridDim.x * blockDim.x) {
        const int c = e >= n ? 1 : 0;
        const int64_t i = e - c * n;
        keys[e] = morton(xs + i * dp, g, lo, hi, d, bits, drop, c) | (uint64_t)c << (bits * d - drop);
        idx[e] = (int32_t)i;
    }
}

// The queries on the refs' grids (their bounds: queries outside them clamp to the edge): their keys as the refs'
// entries have them, by query, and a sort entry each, 2 above the key on grid 0.
__global__ void __launch_bounds__(kThreads) qkeys_kernel(const float *__restrict__ xq, int64_t nq, int d, int dp,
                                                         const uint32_t *__restrict__ lo, const uint32_t *__restrict__ hi,
                                                         int bits, int drop, uint64_t *__restrict__ k0,
                                                         uint64_t *__restrict__ k1, uint64_t *__restrict__ keys,
                                                         int32_t *__restrict__ idx) {
    const Grids g = grids_of(lo, hi, d, bits);
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < 2 * nq; e += (int64_t)gridDim.x * blockDim.x) {
        const int c = e >= nq ? 1 : 0;
        const int64_t q = e - c * nq;
        const uint64_t key = morton(xq + q * dp, g, lo, hi, d, bits, drop, c);
        if (c == 1) {
            k1[q] = key | 1ull << (bits * d - drop);
        } else {
            k0[q] = key;
            keys[q] = key | 2ull << (bits * d - drop);
            idx[q] = (int32_t)q;
        }
    }
}

// float4 index of the v-th 4 features of place k in a curve's coordinates
__host__ __device__ __forceinline__ int64_t coords_at(int64_t k, int v, int v4) {
    return ((k >> 5) * v4 + v) * 32 + (k & 31);
}
__host__ __device__ __forceinline__ int64_t blocks_of(int64_t n) { return (n + 31) / 32; }

// Of each curve (entries [0, n) and [n, 2n) of the sorted order): the points' positions, pos[c n + point], and
// the coordinates in the curve's order, so that the seed kernels' window reads are contiguous: blocks of 32 places,
// in each block 4 features of all 32 after one another (coords_at), 512 bytes for a warp's load of them (by rows of
// dp floats a load touched 4 times as many lines at d = 16).
__global__ void __launch_bounds__(kThreads) place_kernel(const float *__restrict__ xs, int64_t n, int dp,
                                                         const int32_t *__restrict__ order, int32_t *__restrict__ pos,
                                                         float *__restrict__ xs_c) {
    const float4 *src = reinterpret_cast<const float4 *>(xs);
    float4 *dst = reinterpret_cast<float4 *>(xs_c);
    const int v4 = dp / 4;
    const int64_t total = 2 * n * v4, curve = blocks_of(n) * 32 * v4;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t e = t / v4, v = t - e * v4;
        const int64_t i = order[e];
        const int64_t k = e >= n ? e - n : e;
        dst[(e >= n ? curve : 0) + coords_at(k, (int)v, v4)] = src[i * v4 + v];
        if (v == 0) pos[(e >= n ? n : 0) + i] = (int32_t)k;
    }
}

__global__ void __launch_bounds__(kThreads) cross_pos_kernel(const int32_t *__restrict__ order1,
                                                             const int32_t *__restrict__ pos0, int64_t n,
                                                             int32_t *__restrict__ p0_of1) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
        p0_of1[k] = pos0[order1[k]];
}

// Coordinates of place k of a curve.
template <int D>
__device__ __forceinline__ void load_coords(const float4 *__restrict__ xs_c, int64_t k, int v4, float (&r)[(D + 3) / 4 * 4]) {
    const float4 *p = xs_c + coords_at(k, 0, v4);
#pragma unroll
    for (int v = 0; v < (D + 3) / 4; ++v) {
        const float4 t = __ldg(p + 32 * v);
        r[4 * v] = t.x;
        r[4 * v + 1] = t.y;
        r[4 * v + 2] = t.z;
        r[4 * v + 3] = t.w;
    }
}

// Squared distance bits of the ref at place k and the query coordinates qv in the search's exact
// arithmetic: ((r0 - q0)^2 + (r1 - q1)^2) + ..., every step rounded, over the D padded features.
template <int D>
__device__ __forceinline__ uint32_t dist_bits(const float4 *__restrict__ xs_c, int64_t k, int v4, const float (&qv)[D]) {
    float r[(D + 3) / 4 * 4];
    load_coords<D>(xs_c, k, v4, r);
    const float t0 = sub_rn(r[0], qv[0]);
    float d2 = mul_rn(t0, t0);
#pragma unroll
    for (int f = 1; f < D; ++f) {
        const float t = sub_rn(r[f], qv[f]);
        d2 = add_rn(d2, mul_rn(t, t));
    }
    return __float_as_uint(d2);  // NaN bits lie above kInfBits and are never counted
}

// The m-th smallest of the warp's values (each lane holds N; 0xFFFFFFFF = none, NaN bits above kInfBits never
// count), or within kTolBits above it: bisection on the bit patterns until a bound has exactly m values at or
// below it, whose largest is the answer, or the bounds meet; kInfBits when fewer than m values are finite.  Where every
// lane has a value and m <= 32 the largest of the lanes' smallest bounds it from the start.
template <int N>
__device__ __forceinline__ uint32_t mth_smallest_bits(const uint32_t (&v)[N], int m) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    auto count_le = [&](uint32_t bound) -> int {
        int c = 0;
#pragma unroll
        for (int e = 0; e < N; ++e) c += v[e] <= bound ? 1 : 0;
        return (int)__reduce_add_sync(FULL, (unsigned)c);
    };
    uint32_t mn = 0xFFFFFFFFu;
#pragma unroll
    for (int e = 0; e < N; ++e) mn = min(mn, v[e]);
    uint32_t lo = __reduce_min_sync(FULL, mn), hi = __reduce_max_sync(FULL, mn);
    if (m > 32 || hi > kInfBits) {
        if (count_le(kInfBits) < m) return kInfBits;
        hi = kInfBits;
    }
    while (hi - lo > kTolBits) {  // invariant: count_le(hi) >= m; warp-uniform
        const uint32_t mid = lo + ((hi - lo) >> 1);
        const int c = count_le(mid);
        if (c >= m) {
            hi = mid;
            if (c == m) break;
        } else {
            lo = mid + 1;
        }
    }
    uint32_t mx = 0u;  // the largest value at or below hi
#pragma unroll
    for (int e = 0; e < N; ++e) mx = max(mx, v[e] <= hi ? v[e] : 0u);
    return __reduce_max_sync(FULL, mx);
}

// One warp per point (taken in curve-0 order).  Lane values: squared-distance bits of the refs
// j < i in the window [p - W, p + W) of each curve (curve 1 skips refs inside curve 0's window,
// so every ref counts once); 0xFFFFFFFF for the other slots.  The row's seed is the m-th
// smallest value (bisection on the bit patterns, stopped within kTolBits above it), or +inf.
// xs0 / xs1: the coordinates in curve order; p0_of1[k] = curve-0 position of order1[k].
// Bound by the window reads (half of each window is j >= i) and the bisection's counts.  Coordinates by rows -> in blocks
// of 32 places, and a bisection that ends when its count is m, from the lanes' smallest values: 930 -> 807 us (n =
// 434,874, d = 3, two levels), 1,243 -> 989 us (d = 8), 3,734 -> 3,451 us (n = 1M, d = 16, three levels).
template <int D, int VPL>
__global__ void __launch_bounds__(kThreads) seed_kernel(const float4 *__restrict__ xs0,
                                                        const float4 *__restrict__ xs1, int64_t n, int v4, int m, const int32_t *__restrict__ order0,
                                                        const int32_t *__restrict__ order1,
                                                        const int32_t *__restrict__ p0_of1,
                                                        const int32_t *__restrict__ pos1, int combine,
                                                        int64_t row_lo, int64_t row_hi, float *__restrict__ seeds) {
    constexpr int W = VPL * 16;
    const int lane = threadIdx.x & 31;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t k = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; k < n; k += nwarps) {
        const int64_t i = order0[k];
        if (i < row_lo || i >= row_hi) continue;  // another rank's rows (left unset)
        if (i < m) {  // fewer than m earlier points: no bound
            if (lane == 0 && !combine) seeds[i] = __uint_as_float(kInfBits);
            continue;
        }
        float row[(D + 3) / 4 * 4], qv[D];
        load_coords<D>(xs0, k, v4, row);
#pragma unroll
        for (int f = 0; f < D; ++f) qv[f] = row[f];
        uint32_t v[2 * VPL];
#pragma unroll
        for (int t = 0; t < VPL; ++t) {
            const int64_t pk = k - W + lane + 32 * t;
            uint32_t val = 0xFFFFFFFFu;
            if (pk >= 0 && pk < n) {
                const int64_t j = order0[pk];
                if (j < i) val = dist_bits<D>(xs0, pk, v4, qv);
            }
            v[t] = val;
        }
        const int64_t p1 = pos1[i];
#pragma unroll
        for (int t = 0; t < VPL; ++t) {
            const int64_t pk = p1 - W + lane + 32 * t;
            uint32_t val = 0xFFFFFFFFu;
            if (pk >= 0 && pk < n) {
                const int64_t j = order1[pk];
                if (j < i) {
                    const int64_t pj = p0_of1[pk];
                    if (pj < k - W || pj >= k + W) val = dist_bits<D>(xs1, pk, v4, qv);
                }
            }
            v[VPL + t] = val;
        }
        const uint32_t res = mth_smallest_bits<2 * VPL>(v, m);
        if (lane == 0) seeds[i] = combine ? fminf(seeds[i], __uint_as_float(res)) : __uint_as_float(res);
    }
}

// First position in keys[0, n) whose key is >= key (keys ascending).
__device__ __forceinline__ int64_t lower_bound_u64(const uint64_t *__restrict__ keys, int64_t n, uint64_t key) {
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (keys[mid] < key) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Seeds of queries against refs (no prefix rule: every ref counts).  One warp per query, taken
// in curve-0 order (qorder) so that neighbouring warps read the same windows: the query's place
// in each curve of the refs (binary search of its key among the refs' sorted keys), the refs
// within W positions on either side (curve 1 skips refs inside curve 0's window), the m-th
// smallest squared distance in the search's exact arithmetic.
template <int D>
__global__ void __launch_bounds__(kThreads) qseed_kernel(const float4 *__restrict__ xs0,
                                                         const float4 *__restrict__ xs1,
                                                         const uint64_t *__restrict__ keys0s,
                                                         const uint64_t *__restrict__ keys1s, int64_t n_ref,
                                                         const int32_t *__restrict__ p0_of1,
                                                         const float *__restrict__ xq, int64_t n_query,
                                                         const uint64_t *__restrict__ qkey0,
                                                         const uint64_t *__restrict__ qkey1,
                                                         const int32_t *__restrict__ qorder, int dp, int m,
                                                         float *__restrict__ seeds) {
    constexpr int VPL = 8, W = VPL * 16;
    const int lane = threadIdx.x & 31, v4 = dp / 4;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t k = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; k < n_query; k += nwarps) {
        const int64_t q = qorder[k];
        float qv[D];
#pragma unroll
        for (int f = 0; f < D; ++f) qv[f] = xq[q * dp + f];
        const int64_t c0 = lower_bound_u64(keys0s, n_ref, qkey0[q]);
        const int64_t c1 = lower_bound_u64(keys1s, n_ref, qkey1[q]);
        uint32_t v[2 * VPL];
#pragma unroll
        for (int t = 0; t < VPL; ++t) {
            const int64_t pk = c0 - W + lane + 32 * t;
            v[t] = (pk >= 0 && pk < n_ref) ? dist_bits<D>(xs0, pk, v4, qv) : 0xFFFFFFFFu;
        }
#pragma unroll
        for (int t = 0; t < VPL; ++t) {
            const int64_t pk = c1 - W + lane + 32 * t;
            uint32_t val = 0xFFFFFFFFu;
            if (pk >= 0 && pk < n_ref) {
                const int64_t pj = p0_of1[pk];
                if (pj < c0 - W || pj >= c0 + W) val = dist_bits<D>(xs1, pk, v4, qv);
            }
            v[VPL + t] = val;
        }
        const uint32_t res = mth_smallest_bits<2 * VPL>(v, m);
        if (lane == 0) seeds[q] = __uint_as_float(res);
    }
}

struct Layout {
    size_t keys_a, keys_b, idx_a, idx_b, pos, p0of1, xs, bounds, cub, cub_bytes, total;
};

// of n points on two curves, and nq queries sorted with them
Layout layout(int64_t n, int dp, int64_t nq = 0) {
    Layout L{};
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off = align_up(off + bytes, 256);
        return o;
    };
    const size_t entries = 2 * (size_t)n + (size_t)nq;
    L.keys_a = take(entries * 8);
    L.keys_b = take(entries * 8);
    L.idx_a = take(entries * 4);
    L.idx_b = take(entries * 4);
    L.pos = take((size_t)n * 2 * 4);
    L.p0of1 = take((size_t)n * 4);
    L.xs = take((size_t)blocks_of(n) * 32 * 2 * dp * 4);
    L.bounds = take(2 * 256 * 4);
    L.cub_bytes = align_up((size_t)(4u << 20) + entries / 2, 256);  // radix-sort scratch budget
    L.cub = take(L.cub_bytes);
    L.total = off + 256;
    return L;
}

struct SeedArgs {
    const float4 *xs0, *xs1;
    int64_t n;
    int dp, m;
    const int32_t *o0, *o1, *p0of1, *p1;
    int combine;
    int64_t row_lo, row_hi;
    float *seeds;
};

template <int D, int VPL>
void launch_seed(int grid, const SeedArgs &a, cudaStream_t stream) {
    seed_kernel<D, VPL><<<grid, kThreads, 0, stream>>>(a.xs0, a.xs1, a.n, a.dp / 4, a.m, a.o0, a.o1, a.p0of1, a.p1,
                                                       a.combine, a.row_lo, a.row_hi, a.seeds);
}

template <int VPL>
bool dispatch_seed(int D, int grid, const SeedArgs &a, cudaStream_t stream) {
    switch (D) {
        case 1: launch_seed<1, VPL>(grid, a, stream); return true;
        case 2: launch_seed<2, VPL>(grid, a, stream); return true;
        case 3: launch_seed<3, VPL>(grid, a, stream); return true;
        case 4: launch_seed<4, VPL>(grid, a, stream); return true;
        case 5: launch_seed<5, VPL>(grid, a, stream); return true;
        case 6: launch_seed<6, VPL>(grid, a, stream); return true;
        case 7: launch_seed<7, VPL>(grid, a, stream); return true;
        case 8: launch_seed<8, VPL>(grid, a, stream); return true;
        case 12: launch_seed<12, VPL>(grid, a, stream); return true;
        case 16: launch_seed<16, VPL>(grid, a, stream); return true;
        case 20: launch_seed<20, VPL>(grid, a, stream); return true;
        case 24: launch_seed<24, VPL>(grid, a, stream); return true;
    }
    return false;
}

int grid_of(int64_t work) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((work + kThreads - 1) / kThreads, (int64_t)kNumSMsB200 * 8));
}


// The curves of n points (left in a workspace region).
struct Curves {
    const uint64_t *keys0, *keys1;   // sorted keys (curve 1's with a 1 above them)
    const int32_t *order0, *order1;  // the points in each curve's order
    const int32_t *pos0, *pos1;      // and their places in it
    const int32_t *p0of1;            // curve-0 place of curve 1's k-th point
    const float4 *xs0, *xs1;         // coordinates in each curve's order (coords_at)
    const int32_t *qorder;           // the queries in curve-0 order
};
// Both curves, and the queries' order (xq; their keys go to qk0, qk1), come from one radix sort, told apart by the
// bits above the keys.  A pass over 16,000 to 900,000 entries is bound by latency (8 to 14 us), so sorts of their own
// took almost as many times as long: the passes for 16,384 queries in 16,599 refs, d = 18, 161 -> 58 us (the
// whole predict 1.03 -> 0.83 ms), a prefix search of n = 434,874, d = 3 with its n / 8 level 4.97 -> 4.81 ms in all.
nngp_status make_curves(const float *xs, int64_t n, int d, int dp, char *base, const Layout &L, const float *xq, int64_t nq,
                        uint64_t *qk0, uint64_t *qk1, Curves &out, cudaStream_t stream) {
    auto at = [&](size_t off) { return reinterpret_cast<void *>(base + off); };
    uint64_t *keys = static_cast<uint64_t *>(at(L.keys_a));
    int32_t *idx = static_cast<int32_t *>(at(L.idx_a)), *pos = static_cast<int32_t *>(at(L.pos));
    uint32_t *lo = static_cast<uint32_t *>(at(L.bounds)), *hi = lo + 256;
    const int bits = seed::bits(d), drop = seed::key_drop(d);
    const int64_t entries = 2 * n + nq;

    NNGP_CUDA_TRY(cudaMemsetAsync(lo, 0xFF, 256 * 4, stream));
    NNGP_CUDA_TRY(cudaMemsetAsync(hi, 0x00, 256 * 4, stream));
    bounds_kernel<<<grid_of(n), kThreads, 0, stream>>>(xs, n, d, dp, lo, hi);
    NNGP_CUDA_TRY(cudaGetLastError());
    keys_kernel<<<grid_of(2 * n), kThreads, 0, stream>>>(xs, n, d, dp, lo, hi, bits, drop, keys, idx);
    NNGP_CUDA_TRY(cudaGetLastError());
    if (nq > 0) {
        qkeys_kernel<<<grid_of(2 * nq), kThreads, 0, stream>>>(xq, nq, d, dp, lo, hi, bits, drop, qk0, qk1, keys + 2 * n,
                                                               idx + 2 * n);
        NNGP_CUDA_TRY(cudaGetLastError());
    }
    cub::DoubleBuffer<uint64_t> dk(keys, static_cast<uint64_t *>(at(L.keys_b)));
    cub::DoubleBuffer<int32_t> dv(idx, static_cast<int32_t *>(at(L.idx_b)));
    const int end_bit = bits * d - drop + (nq > 0 ? 2 : 1);
    // (a 64-bit count only where 32 bits do not hold it)
    auto sort = [&](void *scratch, size_t &bytes) {
        return entries <= INT_MAX
                   ? cub::DeviceRadixSort::SortPairs(scratch, bytes, dk, dv, (int)entries, 0, end_bit, stream)
                   : cub::DeviceRadixSort::SortPairs(scratch, bytes, dk, dv, entries, 0, end_bit, stream);
    };
    size_t need = 0;
    NNGP_CUDA_TRY(sort(nullptr, need));
    if (need > L.cub_bytes)
        return fail(NNGP_ERR_WORKSPACE,
                    "knn seeds: radix-sort scratch " + std::to_string(need) + " bytes exceeds the budget");
    size_t have = L.cub_bytes;
    NNGP_CUDA_TRY(sort(at(L.cub), have));
    const int32_t *order = dv.Current();
    float *xc = static_cast<float *>(at(L.xs));
    int32_t *p0of1 = static_cast<int32_t *>(at(L.p0of1));
    place_kernel<<<grid_of(2 * n * (dp / 4)), kThreads, 0, stream>>>(xs, n, dp, order, pos, xc);
    NNGP_CUDA_TRY(cudaGetLastError());
    cross_pos_kernel<<<grid_of(n), kThreads, 0, stream>>>(order + n, pos, n, p0of1);
    NNGP_CUDA_TRY(cudaGetLastError());
    out = Curves{dk.Current(), dk.Current() + n, order, order + n, pos, pos + n, p0of1,
                 reinterpret_cast<const float4 *>(xc), reinterpret_cast<const float4 *>(xc) + blocks_of(n) * 32 * (dp / 4),
                 order + 2 * n};
    return NNGP_OK;
}

// One level: seeds of the points [0, n) from the windows of the curves of those points only
// (combine: keep the smaller of the old and the new bound).
// Only the rows [row_lo, row_hi) get seeds (the others are left as they were).
nngp_status run_level(const float *xs, int64_t n, int d, int D, int dp, int m, int W, char *base, const Layout &L,
                      int combine, float *seeds, cudaStream_t stream, Curves &cv, int64_t row_lo, int64_t row_hi) {
    nngp_status st = make_curves(xs, n, d, dp, base, L, nullptr, 0, nullptr, nullptr, cv, stream);
    if (st != NNGP_OK) return st;
    const int grid = (int)std::min<int64_t>((n + kThreads / 32 - 1) / (kThreads / 32), (int64_t)kNumSMsB200 * 16);
    const SeedArgs sa{cv.xs0, cv.xs1, n, dp, m, cv.order0, cv.order1, cv.p0of1, cv.pos1, combine, row_lo, row_hi, seeds};
    const bool ok = W == 128 ? dispatch_seed<8>(D, grid, sa, stream) : dispatch_seed<16>(D, grid, sa, stream);
    if (!ok) return fail(NNGP_ERR_UNSUPPORTED, "knn seeds: no kernel for D = " + std::to_string(D));
    NNGP_CUDA_TRY(cudaGetLastError());
    return NNGP_OK;
}

template <int D>
void launch_qseed(int grid, const float4 *xs0, const float4 *xs1, const uint64_t *k0s, const uint64_t *k1s, int64_t n_ref,
                  const int32_t *p0of1, const float *xq, int64_t nq, const uint64_t *qk0, const uint64_t *qk1,
                  const int32_t *qorder, int dp, int m, float *seeds, cudaStream_t stream) {
    qseed_kernel<D><<<grid, kThreads, 0, stream>>>(xs0, xs1, k0s, k1s, n_ref, p0of1, xq, nq, qk0, qk1, qorder, dp, m,
                                                   seeds);
}

// Refinement levels: prefixes n / 8, n / 64, ... (while at least kMinPoints), run in a second
// workspace region sized for n / 8.
size_t sub_bytes(int64_t n, int dp) { return n / 8 >= kMinPoints ? layout(n / 8, dp).total : 0; }

}  // namespace

size_t workspace_query(int64_t n_ref, int64_t n_query, int dp) {
    if (n_ref < kMinPoints || n_query < 1) return 0;
    return align_up(layout(n_ref, dp, n_query).total, 256) + (size_t)n_query * 16;  // and the queries' keys
}

nngp_status query_seeds(const float *xs_ref, int64_t n_ref, const float *xq, int64_t n_query, int d, int D, int dp,
                        int m, void *ws, size_t ws_bytes, float *seeds, cudaStream_t stream, const int32_t **order0_out,
                        const int32_t **qorder_out) {
    if (n_ref < kMinPoints || n_query < 1 || m < 1 || d < 1 || d > 24 || D < d || dp % 4 != 0 || dp < D)
        return fail(NNGP_ERR_UNSUPPORTED, "knn query seeds: shape outside the seeded search");
    const Layout L = layout(n_ref, dp, n_query);
    if (!ws || ws_bytes < workspace_query(n_ref, n_query, dp))
        return fail(NNGP_ERR_WORKSPACE, "knn query seeds: workspace too small");
    char *base = reinterpret_cast<char *>(align_up(reinterpret_cast<uintptr_t>(ws), 256));
    uint64_t *qk0 = reinterpret_cast<uint64_t *>(base + align_up(L.total, 256) - 256), *qk1 = qk0 + n_query;
    Curves cv{};
    nngp_status st = make_curves(xs_ref, n_ref, d, dp, base, L, xq, n_query, qk0, qk1, cv, stream);
    if (st != NNGP_OK) return st;
    const int grid = (int)std::min<int64_t>((n_query + kThreads / 32 - 1) / (kThreads / 32), (int64_t)kNumSMsB200 * 16);
    switch (D) {
#define NNGP_QS(DD) \
    case DD:                                                                                                        \
        launch_qseed<DD>(grid, cv.xs0, cv.xs1, cv.keys0, cv.keys1, n_ref, cv.p0of1, xq, n_query, qk0, qk1, cv.qorder, dp, m, \
                         seeds, stream);                                                                          \
        break;
        NNGP_QS(1) NNGP_QS(2) NNGP_QS(3) NNGP_QS(4) NNGP_QS(5) NNGP_QS(6) NNGP_QS(7) NNGP_QS(8) NNGP_QS(12) NNGP_QS(16)
        NNGP_QS(20) NNGP_QS(24)
#undef NNGP_QS
        default: return fail(NNGP_ERR_UNSUPPORTED, "knn query seeds: no kernel for D = " + std::to_string(D));
    }
    NNGP_CUDA_TRY(cudaGetLastError());
    if (order0_out) *order0_out = cv.order0;
    if (qorder_out) *qorder_out = cv.qorder;
    return NNGP_OK;
}

size_t workspace(int64_t n, int dp) {
    return n < kMinPoints ? 0 : align_up(layout(n, dp).total, 256) + sub_bytes(n, dp);
}

int window() {
    const char *env = std::getenv("NNGP_KNN_SEED_W");
    if (!env) return 128;
    const int w = std::atoi(env);
    return (w == 0 || w == 128 || w == 256) ? w : 128;
}

nngp_status prefix_seeds(const float *xs, int64_t n, int d, int D, int dp, int m, void *ws, size_t ws_bytes,
                         float *seeds, cudaStream_t stream, const int32_t **order0_out, const int32_t **pos0_out,
                         const uint64_t **keys0_out, int64_t row_lo, int64_t row_hi) {
    const int W = window();
    if (row_hi < 0 || row_hi > n) row_hi = n;
    if (W == 0 || n < kMinPoints || m < 1 || d < 1 || d > 24 || D < d || dp % 4 != 0 || dp < D)
        return fail(NNGP_ERR_UNSUPPORTED, "knn seeds: shape outside the seeded search");
    const Layout L = layout(n, dp);
    if (!ws || ws_bytes < workspace(n, dp)) return fail(NNGP_ERR_WORKSPACE, "knn seeds: workspace too small");
    char *base = reinterpret_cast<char *>(align_up(reinterpret_cast<uintptr_t>(ws), 256));
    Curves cv{};
    nngp_status st = run_level(xs, n, d, D, dp, m, W, base, L, 0, seeds, stream, cv, row_lo, row_hi);
    if (st != NNGP_OK) return st;
    if (order0_out) *order0_out = cv.order0;
    if (pos0_out) *pos0_out = cv.pos0;
    if (keys0_out) *keys0_out = cv.keys0;
    // rows i < n / 8 see few earlier points in the full windows: bound them again from the
    // curves of the prefix alone (any m earlier points bound a row; the smaller bound is kept)
    char *sub = base + align_up(L.total, 256);
    for (int64_t p = n / 8; p >= kMinPoints && p > row_lo; p /= 8) {
        st = run_level(xs, p, d, D, dp, m, W, sub, layout(p, dp), 1, seeds, stream, cv, row_lo, row_hi);
        if (st != NNGP_OK) return st;
    }
    return NNGP_OK;
}

}  // namespace seed
}  // namespace nngp
