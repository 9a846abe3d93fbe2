// Index arithmetic of the f64 env-map lookups, for host and device.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define TPT_HD __host__ __device__ __forceinline__
#else
#define TPT_HD inline
#endif

namespace tpt {

// floor(f) held to 0 .. n, 0 for a NaN: the reference's `as usize` (src/env.rs:
// 92-182).  A cast alone would not do: an f64 NaN casts to INT_MIN on the GPU
// (an f32 one to 0), and a NaN direction is all it takes.
TPT_HD int texel_index(double f, int n) {
    const double g = floor(f);
    return g > 0.0 ? (g < (double)n ? (int)g : n) : 0;
}

}  // namespace tpt
