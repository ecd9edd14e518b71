// Direct neighbour search (knn_direct.cu), used by the dispatcher in knn.cu.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "nngp_b200.h"

namespace nngp {
namespace direct {

constexpr int kMaxNeighbours = 128;  // larger lists take the generic kernel

// Row length (elements) of the scaled, zero-padded point arrays for d features.
inline int row_len(int d) { return (d + 3) / 4 * 4; }

// Exact lists of n_query queries among n_ref refs (rows of row_len(d) scaled elements, 16-byte
// aligned): the contract of knn.cu.  1 <= m <= kMaxNeighbours, T float or double.
template <typename T>
nngp_status search(const T *refs, int64_t n_ref, const T *qs, int64_t n_query, int d, int m, int has_cut, int64_t cut,
                   int32_t *out, cudaStream_t stream);

}  // namespace direct
}  // namespace nngp
