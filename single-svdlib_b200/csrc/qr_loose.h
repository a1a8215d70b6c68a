// When a factorisation's Gram matrix shows that X R^-1 may not be orthonormal
// to rounding.  Free of kernels, so that the bound can be checked on the host.
//
// ||G - I||_F bounds the spectral norm: below 0.5 every singular value of X
// lies in [0.70, 1.23], kappa(X) is below 1.8, and one CholeskyQR pass leaves
// X R^-1 orthonormal to rounding.  The largest entry of G - I does not do: a
// defect a v v^T spread over c = 60 columns changes no entry by more than
// 0.017 a, and kappa is 100 at a = 0.9999.
#pragma once

#include <cuda_runtime.h>

namespace svdb {

// entry (i, j)'s share of ||G - I||_F^2, for a symmetric G given by j >= i
__host__ __device__ inline double loose_term(double g, int i, int j) {
    const double d = i == j ? g - 1.0 : g;
    return j > i ? 2.0 * d * d : j == i ? d * d : 0.0;
}
__host__ __device__ inline bool is_loose(double sum) { return !(sum <= 0.25); }  // NaN is

}  // namespace svdb
