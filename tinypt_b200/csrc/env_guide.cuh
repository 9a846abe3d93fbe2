// Starting brackets for the searches of non-decreasing CDFs (env_guide.cu).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace tpt {

// Equal buckets of the variate a table for CDFs of n entries has: the power of
// two from n, at most 1024 (a variate times it is exact).  0: no table, as an
// entry would not fit 16 bits.
inline int guide_buckets(size_t n) {
    if (n < 2 || n > 65535) return 0;
    int k = 1;
    while ((size_t)k < n && k < 1024) k *= 2;
    return k;
}

// Fills guide[row * (k + 1) + j], j = 0 .. k = guide_buckets(n): the largest lo in
// [0, n - 2] with cdf[row * n + lo] <= j / k * scale (0 if none).  For x = u *
// scale, u in [0, 1), the answer lies between the entries of u's bucket.  The f64
// form's row scales are the differences of row_ends where that is given.
cudaError_t make_guide(const float* cdf, size_t rows, size_t n, uint16_t* guide, cudaStream_t stream);
cudaError_t make_guide(const double* cdf, size_t rows, size_t n, const double* row_ends, double scale, uint16_t* guide,
                       cudaStream_t stream);

}  // namespace tpt
