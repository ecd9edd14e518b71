// Cells of the pruned prefix search (knn_cells.cu): which pivot each point is nearest to, and how far
// a set of points reaches from its pivot towards every other one.  Used by knn_prune.cu.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "nngp_b200.h"

namespace nngp {
namespace cells {

constexpr int kMaxCells = 128;
// Cells are used from this many features and points on.  With fewer features boxes along the curve do as well and
// cells cost partly filled groups (n = 434,874, with against without: uniform d = 5 12.9 / 10.8 ms, d = 6 17.0 / 16.9,
// d = 8 26.8 / 26.4, d = 8 ARD 18.3 / 19.2); with fewer points the groups of a cell are too small (mixture d = 10,
// n = 70,000 4.2 / 3.3 ms; n = 140,000 5.8 / 6.6; d = 16, n = 131,072 5.6 / 6.4, n = 200,000 7.1 / 10.7; d = 24, n =
// 300,000 9.2 / 17.5).  Points that are not clustered pay for the planning and gain little: uniform and normal, d = 9
// to 24, with against without 3 % slower at n = 140,000 (d = 9 4.62 / 4.49 ms), 1 to 2 % at 434,874 and 1 % at 1M;
// points near a 4-dimensional surface 4.67 / 4.17 ms at d = 9, n = 140,000, 30.1 / 35.7 at d = 16, n = 1M, 37.6 / 51.2
// at d = 24, n = 1M.
constexpr int kMinDim = 9;
constexpr int64_t kMinPoints = 131072;

// Cells for n points: 0 where they are not used, else a power of two, about n / 4,096, 32 to kMaxCells.
int count(int64_t n, int d);

struct Cells {
    int K = 0;                       // 0: no cells
    const uint8_t *of = nullptr;     // cell of point i
    const float *pivots = nullptr;   // K rows of dp floats
    const float *dirs = nullptr;     // dirs[(b * d + f) * K + a]: feature f of the unit vector from pivot b to pivot a
    const float *apart = nullptr;    // apart[a * K + b] <= the distance from pivot a to pivot b along that vector
};

size_t workspace(int64_t n, int d);

// Pivots (a few k-means steps on a sample), their directions, and every point's cell.  xs: n scaled points, row
// stride dp.  Any pivots give exact searches; better ones list fewer tiles.
nngp_status build(const float *xs, int64_t n, int d, int dp, void *ws, size_t ws_bytes, Cells *out, cudaStream_t stream);

// Reach of sets of points: set s = points order[off[s] .. off[s + 1]) (off == nullptr: order[128 s .. min(128 (s +
// 1), n))), at most max_sets of them (*n_sets when not null).  home[s] = the cell of its first point, b, and
// for every pivot a != b reach(s, a) >= the largest (x - pivot_b) . dir(b, a) over its points x: stored at
// reach[s * K + a], or with transposed at reach[a * max_sets + s].
nngp_status reach(const Cells &c, const float *xs, int d, int dp, int64_t n, const int32_t *order, const int32_t *off,
                  const int64_t *n_sets, int64_t max_sets, bool transposed, int32_t *home, float *reach,
                  cudaStream_t stream);

}  // namespace cells
}  // namespace nngp
