// Local systems of up to 64 neighbours: 32 / LPP points per warp, LPP lanes per point (local.cu
// has the mathematics).
//
// Lane `sub` of a point's group owns the rows c * LPP + sub, c = 0 .. C - 1 (C = M / LPP), of the
// neighbour block, row i up to column (c + 1) * LPP - 1: with the rows of one class c equally long,
// every loop bound is a compile-time constant and only the diagonal LPP x LPP blocks hold
// entries above the diagonal.  M is the neighbour count rounded up to 16, 32 or 64; rows past it and
// missing neighbours are identity rows.
//
// LPP is M / 2, two rows per lane and one, two or four points per warp, or M, one row per lane (few
// points, many features: rows_per_lane).  Why two rows: with one row per lane a lane computes whole
// rows of a symmetric matrix, twice the fill's and three times the factor's work, and the chain of
// each column (two shuffles, a reciprocal square root, a trip through shared memory) is paid per
// point.  At M = 32 a warp issues 24 fill entries per point instead of 32 and 308 factor FMAs instead
// of 496, and one chain serves two points.  Every value is formed by the same operations in the same
// order with either (sums over the rows by the same butterfly tree), so FP32 systems give the same bits.
//
// Bound by latency: about 3,400 (FP32) and 4,500 (FP64) instructions per point at 2.5 to 3 warps per
// scheduler, each waiting for fixed-latency chains, shared-memory round trips and the gather.
// Measured against one row per lane (one B200): FP32 n = 1,000,000, d = 16, m = 32 with gradient 8.66 ->
// 5.80 ms; FP64 n = 434,874, d = 3 5.11 -> 3.5 ms; FP32 n = 100,000, d = 5, m = 13 0.74 -> 0.17 ms.  Four points per
// warp at M = 32 (8.3 ms in FP32: 255 registers and 6 warps per SM) and everything unrolled
// (6.5 ms) were slower.  The factor in two column blocks instead of one sweep: FP32 5.80 -> 5.52 ms, FP64
// 3.49 -> 3.54 ms.  M = 64 (FP64, kernel values recomputed for the gradient to fit 5 warps per SM): n =
// 20,000, d = 4 ARD, m = 64, two outputs 15.0 ms with one CTA per system -> 1.40 ms.
//
// Shared memory per point (PtLayout): the factor by columns, L[i][k] (i > k) at le[k * lda + i], whose
// unused upper part keeps the squared distances, R[i][k] (k < i) at le[i * lda + k]; the scaled
// coordinates, whose place the fill's kernel values E[i][k] (k < i) take when the gradient needs
// those and the coordinates no more; reciprocal diagonal; b and v.
// Row strides are odd multiples of 16 bytes and a point's block is 16 (mod 128) bytes, so that the
// 16-byte loads of 8 lanes, and of the points of a warp, fall into different banks.
#pragma once

#include <algorithm>

#include "local.cuh"

namespace nngp {

constexpr int kLocalGridPerSm = 8;  // CTAs per SM at most (bounds the partial sums of a launch)

// 16 bytes of TC
template <typename TC> struct Vec16;
template <> struct Vec16<double> {
    static constexpr int N = 2;
    using T = double2;
    __device__ static double get(const double2 &v, int e) { return e == 0 ? v.x : v.y; }
    __device__ static double2 make(const double *p) { return make_double2(p[0], p[1]); }
};
template <> struct Vec16<float> {
    static constexpr int N = 4;
    using T = float4;
    __device__ static float get(const float4 &v, int e) { return e == 0 ? v.x : (e == 1 ? v.y : (e == 2 ? v.z : v.w)); }
    __device__ static float4 make(const float *p) { return make_float4(p[0], p[1], p[2], p[3]); }
};

// C: rows per lane (1 or 2).  Lanes per point of the systems with M rows.
__host__ __device__ constexpr int lanes_per_point(int M, int C) { return M / C; }

// Resident CTAs (of two warps) per SM the registers are budgeted for: FP32 and the 16-row systems 168
// registers, 12 warps per SM; the 32- and 64-row FP64 ones are held to 8 and 5 warps by shared memory, so
// they get the registers they ask for.
template <typename TIn, int M, bool PRED> constexpr int kWarpMinCtas =
    !PRED && (M == 16 || (M == 32 && std::is_same<TIn, float>::value)) ? 6 : 1;

// Elements before row i of the packed kernel values: row i holds its columns k < i, rounded up to 4.
__host__ __device__ inline int packed_row(int i) {
    const int n = i > 0 ? i - 1 : 0, q = n / 4;
    return 8 * q * (q + 1) + 4 * (n % 4) * (q + 1);
}

struct PtLayout {
    int ds, lda;                      // row strides in elements
    size_t le, xs, e, idg, bv, total;  // byte offsets in a point's block, and its size
    // keep_e: the kernel values are kept for the gradient (RBF); in the coordinates' place unless those
    // are needed again (keep_x: per-feature length-scale terms)
    template <typename TC> __host__ __device__ static PtLayout make(int M, int d, bool grad, bool keep_e, bool keep_x) {
        constexpr int EV = 16 / (int)sizeof(TC);
        PtLayout s;
        s.ds = EV * (((d + EV - 1) / EV) | 1);
        s.lda = M + EV;
        const size_t x = (size_t)(M + 1) * s.ds, e = keep_e ? (size_t)packed_row(M) : 0;
        s.le = 0;
        s.xs = (size_t)M * s.lda * sizeof(TC);
        s.e = keep_x ? s.xs + x * sizeof(TC) : s.xs;
        s.idg = s.xs + (keep_x ? x + e : (x > e ? x : e)) * sizeof(TC);
        s.bv = s.idg + (size_t)M * sizeof(TC);
        s.total = s.bv + (grad ? (size_t)2 * M * sizeof(TC) : 0);
        s.total = (s.total + 111) / 128 * 128 + 16;
        return s;
    }
};

// Shared memory of one warp: the blocks of its points (of the larger kind where a kernel solves in
// both precisions), then one gradient accumulator per group.
struct WarpLayout {
    size_t g, total;
    template <bool F32, bool F64>
    __host__ __device__ static WarpLayout make(int M, int C, int d, int n_theta, bool grad, bool keep_e, bool keep_x) {
        const int groups = 32 / lanes_per_point(M, C);
        size_t b = 0;
        if (F32) b = groups * PtLayout::make<float>(M, d, grad, keep_e, keep_x).total;
        if (F64) {
            const size_t q = groups * PtLayout::make<double>(M, d, grad, keep_e, keep_x).total;
            b = q > b ? q : b;
        }
        WarpLayout w;
        w.g = (b + 15) / 16 * 16;
        w.total = (w.g + (size_t)groups * n_theta * 8 + 15) / 16 * 16;
        return w;
    }
};

// Solves the system of point p for each group of LPP lanes (p < 0: the group has none; it runs along).
// Returns false (and commits nothing) for the groups whose FP32 system has a pivot below the FP64
// threshold.  ll_acc: the group's sum, held by its first lane; gacc: the group's gradient sums.
template <typename TC, typename TIn, int M, int C, bool GRAD, bool PRED, bool MATERN>
__device__ __forceinline__ bool solve_points(const LocalArgs &a, const int64_t p, const int lane,
                                             const TIn *__restrict__ x_ref, const TIn *__restrict__ y_ref,
                                             const TIn *__restrict__ x_pt, const TIn *__restrict__ y_pt,
                                             const int32_t *__restrict__ nbr, unsigned char *wsm, double *gacc,
                                             double &ll_acc, TIn *__restrict__ mean, TIn *__restrict__ var,
                                             int32_t *__restrict__ flags) {
    constexpr int LPP = lanes_per_point(M, C);
    using V = Vec16<TC>;
    using VT = typename V::T;
    constexpr int EV = V::N;
    constexpr unsigned FULL = 0xffffffffu;
    constexpr bool STASH = GRAD && !MATERN && M <= 32;  // RBF gradient: reuse the fill's kernel values
    // (opaque, so that addresses and predicates that depend on the lane are formed where they are used
    // instead of being kept in registers, then in local memory, across the loop over the points)
    int lane_here = lane;
    asm volatile("" : "+r"(lane_here));
    const int sub = lane_here & (LPP - 1), grp = lane_here / LPP;
    const Hyp h = hyp_of(a);
    const PtLayout lay = PtLayout::make<TC>(M, a.d, GRAD, STASH, GRAD && a.ard);
    unsigned char *ptsm = wsm + grp * lay.total;
    TC *LE = reinterpret_cast<TC *>(ptsm + lay.le);
    TC *xs = reinterpret_cast<TC *>(ptsm + lay.xs);
    TC *Es = reinterpret_cast<TC *>(ptsm + lay.e);
    TC *idg = reinterpret_cast<TC *>(ptsm + lay.idg);
    TC *bs = reinterpret_cast<TC *>(ptsm + lay.bv), *vs = bs + M;
    constexpr int LDA = M + EV;
    const int d = a.d, ds = lay.ds;
    const bool act = p >= 0;
    auto row_of = [&](int c) { return c * LPP + sub; };
    // sum of one value per row over the point's rows: the tree of a 32-lane butterfly
    auto lanes_sum = [&](TC v) -> TC {
#pragma unroll
        for (int o = LPP / 2; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
        return v;
    };
    auto rows_sum = [&](const TC (&w)[C]) -> TC {
        if constexpr (C == 2) return lanes_sum(add_rn(w[0], w[1]));
        else return lanes_sum(w[0]);
    };
    // f(dc, k0) for every 4 columns k0 .. k0 + 3 of the lower triangle: dc is the class of their rows'
    // diagonal block (a constant once inlined), the rows of the classes c >= dc reach them.  Loops,
    // not unrolled code: a kernel of 4,000 straight instructions waits for its instructions.
    auto for_columns = [&](auto &&f) {
#pragma unroll 1
        for (int k0 = 0; k0 < LPP; k0 += 4) f(0, k0);
        if constexpr (C > 1) {
#pragma unroll 1
            for (int k0 = LPP; k0 < 2 * LPP; k0 += 4) f(1, k0);
        }
    };
    auto store4 = [&](TC *at, const TC (&w)[4]) {
#pragma unroll
        for (int q = 0; q < 4; q += EV) *reinterpret_cast<VT *>(at + q) = V::make(w + q);
    };
    auto load4 = [&](const TC *at, TC (&w)[4]) {
#pragma unroll
        for (int q = 0; q < 4; q += EV) {
            const VT v = *reinterpret_cast<const VT *>(at + q);
#pragma unroll
            for (int e = 0; e < EV; ++e) w[q + e] = V::get(v, e);
        }
    };

    // ---- neighbours of this lane's rows ----------------------------------------------------
    int32_t j[C];
    bool valid[C];
    using Mask = typename std::conditional<(M > 32), unsigned long long, unsigned>::type;
    Mask vmask = 0;  // valid rows of the point
#pragma unroll
    for (int c = 0; c < C; ++c) {
        j[c] = -1;
        if (act && row_of(c) < a.m) {
            j[c] = __ldg(nbr + p * a.m + row_of(c));
            if (j[c] < -1 || (int64_t)j[c] >= a.n_rows) {
                flag_or(flags, NNGP_FLAG_BAD_INDEX);
                j[c] = -1;
            }
        }
        valid[c] = j[c] >= 0;
    }
#pragma unroll
    for (int c = 0; c < C; ++c)
        vmask |= (Mask)((__ballot_sync(FULL, valid[c]) >> (grp * LPP % 32)) & (0xffffffffu >> (32 - LPP))) << (c * LPP);

    // ---- gather scaled coordinates: rows 0..M-1 neighbours, row M the point ------------------
    __syncwarp();
    {
        // 16-byte loads where every row starts on 16 bytes
        constexpr int IV = 16 / (int)sizeof(TIn);
        const TC s0 = (TC)h.inv_ls[0];
        const bool wide = d % IV == 0 && ((reinterpret_cast<uintptr_t>(x_ref) | reinterpret_cast<uintptr_t>(x_pt)) & 15) == 0;
        if (wide) {
            using IVT = typename Vec16<TIn>::T;
            for (int f = 0; f < d; f += IV) {
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    IVT v{};
                    if (valid[c]) v = __ldg(reinterpret_cast<const IVT *>(x_ref + (int64_t)j[c] * d + f));
#pragma unroll
                    for (int e = 0; e < IV; ++e) {
                        const TC s = a.ard ? (TC)h.inv_ls[f + e] : s0;
                        xs[row_of(c) * ds + f + e] = valid[c] ? (TC)Vec16<TIn>::get(v, e) * s : TC(0);
                    }
                }
            }
        } else {
            for (int f = 0; f < d; ++f) {
                const TC s = a.ard ? (TC)h.inv_ls[f] : s0;
#pragma unroll
                for (int c = 0; c < C; ++c)
                    xs[row_of(c) * ds + f] = valid[c] ? (TC)x_ref[(int64_t)j[c] * d + f] * s : TC(0);
            }
        }
        for (int f = sub; f < d; f += LPP)
            xs[M * ds + f] = act ? (TC)x_pt[p * d + f] * (a.ard ? (TC)h.inv_ls[f] : s0) : TC(0);
        if (d % EV) {  // rows are read as whole vectors: their padding adds exact zeros
            const int de = (d + EV - 1) / EV * EV;
            for (int f = d; f < de; ++f)
#pragma unroll
                for (int c = 0; c < C; ++c) xs[row_of(c) * ds + f] = TC(0);
            for (int f = d + sub; f < de; f += LPP) xs[M * ds + f] = TC(0);
        }
    }
    __syncwarp();

    // ---- fill: squared scaled distances, kernel values ----------------------------------------
    // squared distances of this lane's rows (classes >= dc) to the points k0 .. k0 + 3
    const int nv = EV == 4 ? (d + EV - 1) / EV : d / EV;
    auto distances4 = [&](const int dc, const int k0, TC(&q)[C][4]) {
#pragma unroll
        for (int c = dc; c < C; ++c)
#pragma unroll
            for (int u = 0; u < 4; ++u) q[c][u] = TC(0);
#pragma unroll 1
        for (int v = 0; v < nv; ++v) {
            VT xi[C];
#pragma unroll
            for (int c = dc; c < C; ++c) xi[c] = *reinterpret_cast<const VT *>(xs + row_of(c) * ds + v * EV);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const VT xk = *reinterpret_cast<const VT *>(xs + (k0 + u) * ds + v * EV);
#pragma unroll
                for (int c = dc; c < C; ++c)
#pragma unroll
                    for (int e = 0; e < EV; ++e) {
                        const TC t = V::get(xi[c], e) - V::get(xk, e);
                        q[c][u] = fma(t, t, q[c][u]);
                    }
            }
        }
        if (EV == 2 && (d & 1)) {  // FP64, odd d: the last feature alone
#pragma unroll
            for (int c = dc; c < C; ++c) {
                const TC xi = xs[row_of(c) * ds + d - 1];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const TC t = xi - xs[(k0 + u) * ds + d - 1];
                    q[c][u] = fma(t, t, q[c][u]);
                }
            }
        }
    };
    const TC rbf = (TC)h.rbf, cst = (TC)h.cst;
    TC rp[C], kvec[C], ep0[C];  // to the point itself
#pragma unroll
    for (int c = 0; c < C; ++c) {
        rp[c] = TC(0);
        for (int f = 0; f < d; ++f) {
            const TC t = xs[row_of(c) * ds + f] - xs[M * ds + f];
            rp[c] = fma(t, t, rp[c]);
        }
        ep0[c] = rbf * kern_s<MATERN>(a.family, rp[c]);  // kept for the gradient
        kvec[c] = valid[c] ? ep0[c] + cst : TC(0);       // K[p][row]
    }
    for_columns([&](const int dc, const int k0) {
        TC q[C][4];
        distances4(dc, k0, q);
#pragma unroll
        for (int c = dc; c < C; ++c)  // around the diagonal also places of K, which is written below
            if (c > dc || k0 < row_of(c)) store4(LE + row_of(c) * LDA + k0, q[c]);
    });
    __syncwarp();  // the coordinates are read: the kernel values take their place
    TC diag_add[C];
    int e_row[C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
        diag_add[c] = (TC)h.noise + ((int64_t)j[c] < a.alpha_below ? (TC)a.alpha : TC(0));
        e_row[c] = packed_row(row_of(c));
    }
    for_columns([&](const int dc, const int k0) {
        TC q[C][4];
#pragma unroll
        for (int c = dc; c < C; ++c) {
            TC ev[4];
            load4(LE + row_of(c) * LDA + k0, q[c]);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool low = c > dc || row_of(c) > k0 + u;
                const bool vk = (vmask >> (k0 + u)) & 1u;
                const TC e = rbf * kern_s<MATERN>(a.family, low ? q[c][u] : TC(0));
                ev[u] = e;
                TC kv = (valid[c] && vk) ? e + cst : TC(0);
                if (c == dc && row_of(c) == k0 + u) kv = valid[c] ? kv + diag_add[c] : TC(1);
                q[c][u] = kv;
            }
            if (STASH && (c > dc || k0 < row_of(c))) store4(Es + e_row[c] + k0, ev);
        }
        __syncwarp();  // (the diagonal block's rows have read the squared distances beside K's places)
#pragma unroll
        for (int c = dc; c < C; ++c)
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (c > dc || row_of(c) >= k0 + u) LE[(k0 + u) * LDA + row_of(c)] = q[c][u];
    });
    __syncwarp();
    const TC kpp = rbf + cst + (TC)h.noise + (PRED ? TC(0) : (TC)a.alpha);

    // ---- Cholesky of the neighbour block fused with l = L^-1 k and the first output's z = L^-1 y ----
    // One block of LPP columns at a time, in registers: the earlier blocks' columns are taken off it
    // (from shared memory), then its own columns are factored right-looking.  Every entry sees the
    // columns in ascending order, as in one right-looking sweep, with a third fewer registers.
    // A row's own results (its pivot's reciprocal, l, z, b, v) are formed once after the loops: the
    // running value of a row stops changing at its own step.
    const bool weights = PRED && a.weights_out;
    TC yv[C];
#pragma unroll
    for (int c = 0; c < C; ++c) yv[c] = (!weights && valid[c]) ? (TC)y_ref[(int64_t)j[c] * a.ydim] : TC(0);
    TC minpiv = TC(3.0e38);
    TC ss = TC(0);
    auto factor_block = [&](const int dc) {
        TC r[C][LPP];  // columns dc * LPP .. of the rows of the classes >= dc (past the diagonal: unused values)
        const int k1 = dc * LPP;
#pragma unroll
        for (int c = dc; c < C; ++c)
#pragma unroll
            for (int q = 0; q < LPP; ++q) r[c][q] = LE[(k1 + q) * LDA + row_of(c)];
        __syncwarp();
#pragma unroll 2
        for (int k = 0; k < k1; ++k) {
            const TC *col = LE + k * LDA;
            TC own[C];
#pragma unroll
            for (int c = dc; c < C; ++c) own[c] = -col[row_of(c)];
#pragma unroll
            for (int q = 0; q < LPP; q += EV) {
                const VT v = *reinterpret_cast<const VT *>(col + k1 + q);
#pragma unroll
                for (int e = 0; e < EV; ++e)
#pragma unroll
                    for (int c = dc; c < C; ++c) r[c][q + e] = fma(own[c], V::get(v, e), r[c][q + e]);
            }
        }
#pragma unroll
        for (int sk = 0; sk < LPP; ++sk) {
            const TC piv = __shfl_sync(FULL, r[dc][sk], sk, LPP);
            minpiv = fmin(minpiv, piv);
            const TC inv = drsqrt<TC>(piv);  // 1 / L_kk
            const TC lk = __shfl_sync(FULL, kvec[dc], sk, LPP) * inv;
            const TC zk = __shfl_sync(FULL, yv[dc], sk, LPP) * inv;
            if (sub == sk) idg[k1 + sk] = inv;
            TC *col = LE + (k1 + sk) * LDA;
#pragma unroll
            for (int c = dc; c < C; ++c) {
                r[c][sk] = r[c][sk] * inv;  // L_ik
                if (c > dc || sub > sk) {
                    kvec[c] = fma(-r[c][sk], lk, kvec[c]);
                    yv[c] = fma(-r[c][sk], zk, yv[c]);
                    col[row_of(c)] = r[c][sk];
                }
            }
            ss = fma(lk, lk, ss);
            __syncwarp();
            if (sk + 1 < LPP) {
#pragma unroll
                for (int q = (sk + 1) / EV * EV; q < LPP; q += EV) {
                    const VT v = *reinterpret_cast<const VT *>(col + k1 + q);
#pragma unroll
                    for (int e = 0; e < EV; ++e) {
                        if (q + e <= sk) continue;
#pragma unroll
                        for (int c = dc; c < C; ++c) r[c][q + e] = fma(-r[c][sk], V::get(v, e), r[c][q + e]);
                    }
                }
            }
        }
    };
    factor_block(0);
    if constexpr (C > 1) factor_block(1);
    const TC s2 = kpp - ss;
    bool ok = true;
    if constexpr (std::is_same<TC, float>::value)
        ok = minpiv >= (TC)h.pivot_abs && s2 >= (TC)h.pivot_abs;  // NaN-safe
    if (act && ok && (!(minpiv > TC(0)) || !(s2 > TC(0)))) flag_or(flags, NNGP_FLAG_NOT_PD);
    __syncwarp();  // the reciprocal diagonal is visible
    TC l_own[C];
#pragma unroll
    for (int c = 0; c < C; ++c) l_own[c] = kvec[c] * idg[row_of(c)];
    const bool commit = act && ok;

    // backward solve of right-hand sides held by rows: w <- L^-T w (the factor read from its
    // columns in shared memory, four rows at a time)
    auto backward = [&](auto &...w) {
#pragma unroll 1
        for (int k0 = M - 4; k0 >= 0; k0 -= 4) {
            TC iv[4], lv[C][4];
            load4(idg + k0, iv);
#pragma unroll
            for (int c = 0; c < C; ++c) load4(LE + row_of(c) * LDA + k0, lv[c]);
#pragma unroll
            for (int u = 3; u >= 0; --u) {
                const int k = k0 + u;
                auto step = [&](TC(&b)[C]) {
                    const TC bc = k0 < LPP ? b[0] : b[C - 1];
                    const TC bk = __shfl_sync(FULL, bc, k & (LPP - 1), LPP) * iv[u];
#pragma unroll
                    for (int c = 0; c < C; ++c)
                        if (row_of(c) < k) b[c] = fma(-lv[c][u], bk, b[c]);
                };
                (step(w), ...);
            }
        }
        auto own = [&](TC(&b)[C]) {
#pragma unroll
            for (int c = 0; c < C; ++c) b[c] = b[c] * idg[row_of(c)];
        };
        (own(w), ...);
    };

    if (PRED && weights) {
        // conditioning weights w = L^-T l = K_nn^-1 k and the variance term s2 (no outputs yet:
        // the full-conditioning recursion combines them with earlier predictions)
        backward(l_own);
        if (commit) {
#pragma unroll
            for (int c = 0; c < C; ++c)
                if (row_of(c) < a.m) mean[p * a.m + row_of(c)] = (TIn)l_own[c];
            if (sub == 0) var[p] = (TIn)s2;
        }
        return ok;
    }

    // ---- outputs -------------------------------------------------------------------------------
    TC zw[C];
#pragma unroll
    for (int c = 0; c < C; ++c) zw[c] = TC(0);
    TC wsum = TC(0);
    double ll = 0.0;
    for (int o = 0; o < a.ydim; ++o) {
        if (o > 0) {
#pragma unroll
            for (int c = 0; c < C; ++c) yv[c] = valid[c] ? (TC)y_ref[(int64_t)j[c] * a.ydim + o] : TC(0);
#pragma unroll 4
            for (int k = 0; k < M; ++k) {
                const TC yc = k < LPP ? yv[0] : yv[C - 1];
                const TC zk = __shfl_sync(FULL, yc, k & (LPP - 1), LPP) * idg[k];
#pragma unroll
                for (int c = 0; c < C; ++c)
                    if (row_of(c) > k) yv[c] = fma(-LE[k * LDA + row_of(c)], zk, yv[c]);
            }
        }
        TC z_own[C], lz[C];
#pragma unroll
        for (int c = 0; c < C; ++c) {
            z_own[c] = yv[c] * idg[row_of(c)];
            lz[c] = mul_rn(l_own[c], z_own[c]);
        }
        const TC mu = rows_sum(lz);
        if (PRED) {
            if (commit && sub == 0) mean[p * a.ydim + o] = (TIn)mu;
        } else {
            const TC res = (act ? (TC)y_pt[p * a.ydim + o] : TC(0)) - mu;
            const double rd = (double)res, sd = (double)s2;
            ll += -0.5 * rd * rd / sd - 0.5 * log(sd) - kHalfLog2Pi;
            if (GRAD) {
                const TC rs = res / s2;
#pragma unroll
                for (int c = 0; c < C; ++c) zw[c] = fma(rs, z_own[c], zw[c]);
                wsum += (res * rs - TC(1)) / (TC(2) * s2);
            }
        }
    }
    if (PRED) {
        if (commit && sub == 0) var[p] = (TIn)s2;
        return ok;
    }
    if (!GRAD) {
        if (commit && sub == 0) ll_acc += ll;
        return ok;
    }

    // ---- adjoint: b = L^-T l, v = L^-T zw ------------------------------------------------------
    backward(l_own, zw);
    TC(&b_own)[C] = l_own;
    TC(&v_own)[C] = zw;
#pragma unroll
    for (int c = 0; c < C; ++c) {
        bs[row_of(c)] = b_own[c];
        vs[row_of(c)] = v_own[c];
    }
    __syncwarp();
    TC g_amp[C], g_cst[C], g_noise[C], g_iso[C];
#pragma unroll
    for (int c = 0; c < C; ++c) g_amp[c] = g_cst[c] = g_noise[c] = g_iso[c] = TC(0);
    for_columns([&](const int dc, const int k0) {
        TC bk[4], vk[4], q[C][4];
        load4(bs + k0, bk);
        load4(vs + k0, vk);
#pragma unroll
        for (int c = dc; c < C; ++c) load4(LE + row_of(c) * LDA + k0, q[c]);
#pragma unroll
        for (int c = dc; c < C; ++c) {
            TC ev[4];
            if (STASH && (c > dc || k0 < row_of(c))) load4(Es + e_row[c] + k0, ev);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int k = k0 + u;
                const bool low = c > dc || row_of(c) > k, own = c == dc && row_of(c) == k;
                const TC rk = low ? q[c][u] : TC(0);  // past the diagonal there is no distance
                // (roundings spelled out, here and below, so that no compiler's choice of fused operations
                // changes the bits)
                const TC bv = fma(v_own[c], bk[u], mul_rn(b_own[c], vk[u]));
                const TC G = fma(mul_rn(wsum, b_own[c]), bk[u], TC(-0.5) * bv);
                const TC wgt = low ? TC(2) : (own ? TC(1) : TC(0));
                const TC s = STASH ? TC(0) : kern_s<MATERN>(a.family, rk);
                const TC gw = wgt * G;
                const TC ge = gw * (STASH ? (low ? ev[u] : (own ? rbf : TC(0))) : rbf * s);
                const TC gl = MATERN ? gw * (rbf * kern_g<MATERN>(a.family, rk, s)) : ge;
                g_amp[c] = add_rn(g_amp[c], ge);
                g_cst[c] += gw;
                if (!a.ard) g_iso[c] = fma(gl, rk, g_iso[c]);
                if (own && valid[c]) g_noise[c] += G;
                ev[u] = gl;
            }
            // kept for the per-feature length-scale terms (0 above the diagonal)
            if (a.ard) store4(LE + row_of(c) * LDA + k0, ev);
        }
    });
    // pair (p, row), weight 2, and (p, p)
    TC gpl[C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
        const TC Gp = valid[c] ? TC(0.5) * v_own[c] - mul_rn(wsum, b_own[c]) : TC(0);
        const TC sp = MATERN ? kern_s<MATERN>(a.family, rp[c]) : TC(0);
        const TC gpe = TC(2) * Gp * (MATERN ? rbf * sp : ep0[c]);
        gpl[c] = MATERN ? TC(2) * Gp * (rbf * kern_g<MATERN>(a.family, rp[c], sp)) : gpe;
        g_amp[c] = add_rn(g_amp[c], gpe);
        g_cst[c] += TC(2) * Gp;
        g_iso[c] = fma(gpl[c], rp[c], g_iso[c]);
    }
    const double amp_t = (double)rows_sum(g_amp) + (double)wsum * h.rbf;
    const double cst_t = (double)rows_sum(g_cst) + (double)wsum;
    const double noi_t = (double)rows_sum(g_noise) + (double)wsum;
    const double iso_t = (double)rows_sum(g_iso);
    if (commit && sub == 0) {
        ll_acc += ll;
        if (a.idx_rbf >= 0) gacc[a.idx_rbf] += amp_t;
        if (a.idx_const >= 0) gacc[a.idx_const] += h.cst * cst_t;
        if (a.idx_noise >= 0) gacc[a.idx_noise] += h.noise * noi_t;
        if (a.idx_ls >= 0 && !a.ard) gacc[a.idx_ls] += iso_t;
    }
    if (a.idx_ls >= 0 && a.ard) {
        // per feature: sum over the pairs of gl * t_f^2
        const int nf = (d + EV - 1) / EV;
#pragma unroll 1
        for (int v = 0; v < nf; ++v) {
            VT xi[C];
            TC acc[EV][C];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                xi[c] = *reinterpret_cast<const VT *>(xs + row_of(c) * ds + v * EV);
#pragma unroll
                for (int e = 0; e < EV; ++e) acc[e][c] = TC(0);
            }
            auto pair = [&](int c, const VT &xk, TC g) {
#pragma unroll
                for (int e = 0; e < EV; ++e) {
                    const TC t = V::get(xi[c], e) - V::get(xk, e);
                    acc[e][c] = fma(g * t, t, acc[e][c]);
                }
            };
            for_columns([&](const int dc, const int k0) {
                TC g[C][4];
#pragma unroll
                for (int c = dc; c < C; ++c) load4(LE + row_of(c) * LDA + k0, g[c]);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const VT xk = *reinterpret_cast<const VT *>(xs + (k0 + u) * ds + v * EV);
#pragma unroll
                    for (int c = dc; c < C; ++c) pair(c, xk, g[c][u]);
                }
            });
            const VT xp = *reinterpret_cast<const VT *>(xs + M * ds + v * EV);
#pragma unroll
            for (int c = 0; c < C; ++c) pair(c, xp, gpl[c]);
#pragma unroll
            for (int e = 0; e < EV; ++e) {
                const double s = (double)rows_sum(acc[e]);
                if (commit && sub == 0 && v * EV + e < d) gacc[a.idx_ls + v * EV + e] += s;
            }
        }
    }
    return ok;
}

// Sum of the groups' and warps' totals in a fixed order: block_out[0 .. n_theta] of this CTA.
template <int GROUPS>
__device__ __forceinline__ void write_partials(const LocalArgs &a, bool grad, const unsigned char *smem, size_t warp_bytes,
                                               size_t g_off, double ll_acc, int sub, int grp, double *block_out) {
    __shared__ double red[4 * GROUPS];
    const int warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    if (sub == 0) red[warp * GROUPS + grp] = ll_acc;
    __syncthreads();
    const int nt = 1 + (grad ? a.n_theta : 0);
    double *o = block_out + (int64_t)blockIdx.x * nt;
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < warps * GROUPS; ++w) s += red[w];
        o[0] = s;
    }
    if (grad) {
        for (int t = threadIdx.x; t < a.n_theta; t += blockDim.x) {
            double s = 0.0;
            for (int w = 0; w < warps; ++w)
                for (int g = 0; g < GROUPS; ++g)
                    s += reinterpret_cast<const double *>(smem + w * warp_bytes + g_off)[g * a.n_theta + t];
            o[1 + t] = s;
        }
    }
}

// The fit step (PRED false) and predict.  Fit-step systems of FP32 inputs that need FP64 are marked
// for local_redo_kernel; predict solves them in place.
template <typename TIn, int M, int C, bool GRAD, bool PRED, bool MATERN>
__global__ void __launch_bounds__(64, (kWarpMinCtas<TIn, M, PRED>)) local_warp_kernel(const __grid_constant__ LocalArgs a,
                                                         const TIn *__restrict__ x_ref, const TIn *__restrict__ y_ref,
                                                         const TIn *__restrict__ x_pt, const TIn *__restrict__ y_pt,
                                                         const int32_t *__restrict__ nbr,
                                                         double *__restrict__ block_out, TIn *__restrict__ mean,
                                                         TIn *__restrict__ var, int32_t *__restrict__ flags) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using T1 = typename std::conditional<(M > 32), double, TIn>::type;  // the first attempt's precision
    constexpr bool F32 = std::is_same<T1, float>::value;
    constexpr int LPP = lanes_per_point(M, C), GROUPS = 32 / LPP;
    const WarpLayout lay = WarpLayout::make<F32, !F32 || PRED>(M, C, a.d, a.n_theta, GRAD,
                                                              GRAD && !MATERN && M <= 32, GRAD && a.ard);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int sub = lane & (LPP - 1), grp = lane / LPP;
    unsigned char *wsm = smem_raw + warp * lay.total;
    double *gacc = reinterpret_cast<double *>(wsm + lay.g) + grp * a.n_theta;
    for (int t = sub; t < a.n_theta; t += LPP) gacc[t] = 0.0;
    __syncwarp();
    double ll_acc = 0.0;
    unsigned long long n_fp64 = 0;
    const int64_t step = (int64_t)gridDim.x * warps * GROUPS;
    for (int64_t p0 = ((int64_t)blockIdx.x * warps + warp) * GROUPS; p0 < a.n_points; p0 += step) {
        const int64_t p = p0 + grp < a.n_points ? p0 + grp : -1;
        const bool ok = solve_points<T1, TIn, M, C, GRAD, PRED, MATERN>(a, p, lane, x_ref, y_ref, x_pt, y_pt, nbr, wsm,
                                                                     gacc, ll_acc, mean, var, flags);
        if constexpr (F32) {
            const bool bad = p >= 0 && !ok;
            if (bad && sub == 0) ++n_fp64;
            if constexpr (!PRED) {
                if (bad && sub == 0) atomicOr(a.redo_bits + (p >> 5), 1u << (p & 31));
            } else {
                if (__any_sync(0xffffffffu, bad))
                    solve_points<double, TIn, M, C, GRAD, PRED, MATERN>(a, bad ? p : -1, lane, x_ref, y_ref, x_pt, y_pt,
                                                                     nbr, wsm, gacc, ll_acc, mean, var, flags);
            }
        }
    }
    if (F32 && n_fp64 > 0) {
        flag_or(flags, NNGP_FLAG_FP64_FALLBACK);
        if (a.fp64_count) atomicAdd(a.fp64_count, n_fp64);
    }
    if (PRED) return;
    write_partials<GROUPS>(a, GRAD, smem_raw, lay.total, lay.g, ll_acc, sub, grp, block_out);
}

// FP64 re-solve of the fit-step systems the FP32 kernel marked; the points of a 32-point word go to
// one warp, words to warps in a fixed order, so the per-CTA partials are deterministic for a given
// launch shape.
template <int M, bool GRAD, bool MATERN>
__global__ void __launch_bounds__(64, (kWarpMinCtas<double, M, false>)) local_redo_kernel(const __grid_constant__ LocalArgs a,
                                                         const float *__restrict__ x_ref, const float *__restrict__ y_ref,
                                                         const float *__restrict__ x_pt, const float *__restrict__ y_pt,
                                                         const int32_t *__restrict__ nbr,
                                                         double *__restrict__ block_out, int32_t *__restrict__ flags) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int C = 2, LPP = lanes_per_point(M, C), GROUPS = 32 / LPP;
    const WarpLayout lay = WarpLayout::make<false, true>(M, C, a.d, a.n_theta, GRAD,
                                                        GRAD && !MATERN && M <= 32, GRAD && a.ard);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int sub = lane & (LPP - 1), grp = lane / LPP;
    unsigned char *wsm = smem_raw + warp * lay.total;
    double *gacc = reinterpret_cast<double *>(wsm + lay.g) + grp * a.n_theta;
    for (int t = sub; t < a.n_theta; t += LPP) gacc[t] = 0.0;
    __syncwarp();
    double ll_acc = 0.0;
    const int64_t words = (a.n_points + 31) / 32;
    for (int64_t w = (int64_t)blockIdx.x * warps + warp; w < words; w += (int64_t)gridDim.x * warps) {
        uint32_t bits = a.redo_bits[w];
        while (bits) {
            int64_t p = -1;
            for (int g = 0; g < GROUPS && bits; ++g) {
                if (g == grp) p = w * 32 + (__ffs(bits) - 1);
                bits &= bits - 1;
            }
            solve_points<double, float, M, C, GRAD, false, MATERN>(a, p, lane, x_ref, y_ref, x_pt, y_pt, nbr, wsm, gacc,
                                                                ll_acc, static_cast<float *>(nullptr),
                                                                static_cast<float *>(nullptr), flags);
        }
    }
    write_partials<GROUPS>(a, GRAD, smem_raw, lay.total, lay.g, ll_acc, sub, grp, block_out);
}

// ---- host side: one launcher per kernel family (local_fit32.cu, local_fit64.cu, local_pred.cu) ------
// Warps per CTA and CTAs of a launch of `need_warps` warps: two warps per CTA (one when their shared
// memory does not fit), as many CTAs as the SMs hold at once (each warp then strides over equal
// shares of the points), at most kLocalGridPerSm per SM.
struct WarpLaunch {
    int warps = 1, grid = 1;
    size_t smem = 0;
};
nngp_status warp_launch(const void *fn, size_t warp_bytes, int64_t need_warps, int grid_limit, WarpLaunch *out);

inline int warp_rows(int m) { return m <= 16 ? 16 : (m <= 32 ? 32 : 64); }

// Rows per lane of a launch: two, or one
//   * for few points, where the length of a warp's program is the time: up to 7 points per SM at M = 32, 22 at M = 16,
//     which one-row warps do in one wave (one against two, us: FP64 d = 18, m = 32 log-likelihood of 300 points
//     25.5 / 31.5, of 1,000 28.7 / 30.9, of 1,200 39.9 / 33.8; FP32 d = 28 with gradient of 1,000 36.6 / 41.0; FP64
//     d = 18, m = 16 log-likelihood of 3,300 24.6 / 28.6, of 4,000 32.8 / 28.8; FP64 gradients at m <= 16 gain nothing
//     from 2,400 points on and lose up to 8 %);
//   * for long rows, whose coordinates leave shared memory for few warps, so that a warp should hold few points: FP64
//     log-likelihood of 30,000 points, m = 32, d = 128 2,049 / 3,413, d = 40 602 / 671, d = 28 496 / 469; FP32 with
//     gradient d = 128 820 / 1,046, d = 64 1.04 times slower; m = 8 FP64 predict d = 28 0.86 of the time, d = 18 equal.
// M = 64 has two.
int rows_per_lane(int M, int d, int64_t n_points, bool f32, bool pred);

// *parts: CTAs of the launch (the partial sums in block_out)
template <typename TIn>
nngp_status launch_fit(const LocalArgs &a, bool grad, const TIn *x_ref, const TIn *y_ref, const TIn *x_pt,
                       const TIn *y_pt, const int32_t *nbr, double *block_out, int grid_limit, int *parts,
                       int32_t *flags, cudaStream_t stream);
nngp_status launch_redo(const LocalArgs &a, bool grad, const float *x_ref, const float *y_ref, const float *x_pt,
                        const float *y_pt, const int32_t *nbr, double *block_out, int grid_limit, int *parts,
                        int32_t *flags, cudaStream_t stream);
template <typename TIn>
nngp_status launch_predict(const LocalArgs &a, const TIn *x_ref, const TIn *y_ref, const TIn *x_pt,
                           const int32_t *nbr, TIn *mean, TIn *var, int32_t *flags, cudaStream_t stream);

}  // namespace nngp
