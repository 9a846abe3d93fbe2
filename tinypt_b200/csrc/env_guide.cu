// Starting brackets of the env map's CDF searches (guide tables: Chen and Asau,
// 1974), made on the device from the CDFs that scene creation has uploaded.  A
// 1024x512 map's tables of both forms hold a million entries: 7 ms on the host,
// under 0.1 here.
#include "env_guide.cuh"

namespace tpt {
namespace {

// Entry j of row r: the answer of the search (env.rs:185-197) for x = j / k *
// scale, the search itself.
template <class T>
__global__ void k_guide(const T* __restrict__ cdf, size_t n, const T* __restrict__ row_ends, T scale, int k,
                        size_t entries, uint16_t* __restrict__ guide) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= entries) return;
    const size_t r = i / (size_t)(k + 1), j = i - r * (size_t)(k + 1);
    if (row_ends) {
        const T d = row_ends[r + 1] - row_ends[r];
        scale = d > (T)0 ? d : (T)0;
    }
    const T x = (T)j / (T)k * scale;
    const T* c = cdf + r * n;
    size_t lo = 0, hi = n - 1;
    while (lo + 1 < hi) {
        const size_t mid = (lo + hi) / 2;
        if (c[mid] <= x) lo = mid;
        else hi = mid;
    }
    guide[i] = (uint16_t)lo;
}

template <class T>
cudaError_t launch(const T* cdf, size_t rows, size_t n, const T* row_ends, T scale, uint16_t* guide, cudaStream_t s) {
    const int k = guide_buckets(n);
    const size_t entries = rows * (size_t)(k + 1);
    k_guide<T><<<(unsigned)((entries + 255) / 256), 256, 0, s>>>(cdf, n, row_ends, scale, k, entries, guide);
    return cudaGetLastError();
}

}  // namespace

cudaError_t make_guide(const float* cdf, size_t rows, size_t n, uint16_t* guide, cudaStream_t stream) {
    return launch<float>(cdf, rows, n, nullptr, 1.0f, guide, stream);
}
cudaError_t make_guide(const double* cdf, size_t rows, size_t n, const double* row_ends, double scale, uint16_t* guide,
                       cudaStream_t stream) {
    return launch<double>(cdf, rows, n, row_ends, scale, guide, stream);
}

}  // namespace tpt
