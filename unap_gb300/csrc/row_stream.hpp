// Products and residuals over large levels (implemented in row_stream.cu).
#pragma once

#include "kernels.hpp"

namespace unapgpu {

// Levels of at least this many rows, of up to 8 entries as a rule (!wide), go
// through the kernels below: each warp of a grid that just fills the GPU then
// has several slices to pipeline.  FP64 product and residual, us, a thread a
// row against here: 13.4/16.0 and 14.4/14.3 at 64^3, 41.1/46.4 and 33.8/35.1
// at 100^3.  FP32 products, bound by memory alone: 14.0 and 14.5 at 100^3, 52
// and 51 at 160^3, 237 and 226 at 256^3.  Wide rows lose (a Chebyshev step of
// 16-entry rows 48 against 99): twice the registers leave too few warps.
constexpr int kStreamRows64 = 1 << 19;
constexpr int kStreamRows32 = 1 << 22;
// A dot product whose partial sums go by more than 256 rows (maxBlocks) stays
// with spmv_kernel.
template <class T>
bool row_streams(const Rows<T>& A, const RSpec& red);

// y = A x and, with a reduction spec, y.dotWith (k_spmv)
template <class T>
void stream_spmv(const Exec& ex, const Rows<T>& A, const T* x, T* y, const T* dotWith, RSpec red,
                 Gate g, bool fused);
// y = A x with y in the order that perm gives
template <class T>
void stream_spmv_reference(const Exec& ex, const Rows<T>& A, const int* perm, const T* x, T* y);
// r = b - A x (k_residual without a reduction)
template <class T>
void stream_residual(const Exec& ex, const Rows<T>& A, const T* x, const T* b, T* r, Gate g);

}  // namespace unapgpu
