// Dense inverse of a sparse symmetric diagonally dominant level by a block
// sweep in nested-dissection order.
#pragma once

#include <cuda_runtime.h>

#include <functional>

#include "kernels.cuh"

namespace fvm {
namespace dev {

// a: the level in SELL-32 (rowSlice: a row's slice), 1 <= n <= 4096; flags:
// one device int, set when a row is not diagonally dominant (bit 0, relative
// slack 1e-8) or an entry not symmetric to a relative 1e-12 (bit 1).
void dominant_symmetric_check(const SellView<double>& a, const int* rowSlice, int* flags, cudaStream_t st);

// Points of a coarse level's rows, x[nc], y[nc], z[nc]: the mean over each
// row's fine rows (c2fRow, c2fCol) of their points (finePoints, nFine each)
// or, fineXyz given, of the cells' (3 per cell; fineCell: a fine row's cell).
void coarse_points(int nc, const int* c2fRow, const int* c2fCol, const int* fineCell, const double* fineXyz, int nFine,
                   const float* finePoints, float* points, cudaStream_t st);

// The inverse, n x n row-major in a's row numbering, to out64 or (out64
// null) in FP32 to outF with rows inverse_f32_stride(n) apart. alloc gives device memory that lives until the
// stream has finished; *status (device, 0 on entry) becomes 1 when a pivot
// is exactly zero. points (may be null): the rows' points, which only shape
// the order of elimination. The order of elimination is read back to the host (one
// synchronisation of the stream), the sweep itself is asynchronous.
void inverse_symmetric(const SellView<double>& a, const int* rowSlice, const float* points, double* out64, float* outF,
                       int* status, const std::function<void*(size_t)>& alloc, cudaStream_t st);

}  // namespace dev
}  // namespace fvm
