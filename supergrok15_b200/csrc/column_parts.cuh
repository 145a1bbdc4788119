// Fixed-order sum of the per-CTA partial rows of a reduction: out[c] = sum_p partial[p][c].  A CTA owns 32 columns; warp w adds the rows
// w, w + 32, ... (four loads in flight) and the 32 sub-sums are added in warp order; in fp64, since the partial rows are few and
// cancel.  One thread per column walked up to 1,700 rows behind one another: 118 us for the scan adjoint, 13 to 29 us for the routing,
// GRU and expert gradients.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace sg {

__device__ __forceinline__ float column_parts_sum(const float* __restrict__ partial, int64_t first, int64_t last, int ng, int c) {
    __shared__ double sh[32][33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double t = 0;
    if (c < ng) {
        int64_t p = first + w;
        for (; p + 96 < last; p += 128) {
            float v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = partial[(p + 32 * u) * ng + c];
#pragma unroll
            for (int u = 0; u < 4; ++u) t += v[u];
        }
        for (; p < last; p += 32) t += partial[p * ng + c];
    }
    sh[w][lane] = t;
    __syncthreads();
    t = 0;
    if (w == 0)
#pragma unroll
        for (int k = 0; k < 32; ++k) t += sh[k][lane];
    return (float)t;                                      // valid in warp 0
}

namespace {
__global__ void __launch_bounds__(1024) column_parts_kernel(const float* __restrict__ partial, int parts, int ng, float* __restrict__ out) {
    const int c = blockIdx.x * 32 + (threadIdx.x & 31);
    const float t = column_parts_sum(partial, 0, parts, ng, c);
    if (threadIdx.x < 32 && c < ng) out[c] = t;
}
}  // namespace

}  // namespace sg
