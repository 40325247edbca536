// The last step of column sums (dB), inside the kernels that finish a filter gradient.
#pragma once
#include <cuda_runtime.h>

namespace aether {

// out[c] = sum over blocks of part[block][C] for the eight columns of CTA `cta` (256 threads): 32 lanes per column, so
// the serial chains are short, combined in fixed order.
__device__ __forceinline__ void finish_columns(const float* __restrict__ part, int nblocks, int C, float* __restrict__ out, int cta,
                                               float (*red)[8]) {
    const int cl = threadIdx.x & 7, lane = threadIdx.x >> 3;
    const int c = cta * 8 + cl;
    float s = 0.f;
    if (c < C) {
        constexpr int U = 8;
        for (int b = lane; b < nblocks; b += 32 * U) {
            float v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) v[u] = b + 32 * u < nblocks ? part[(size_t)(b + 32 * u) * C + c] : 0.f;
#pragma unroll
            for (int u = 0; u < U; ++u) s += v[u];
        }
    }
    red[lane][cl] = s;
    __syncthreads();
    if (lane == 0 && c < C) {
        float t = 0.f;
#pragma unroll
        for (int l = 0; l < 32; ++l) t += red[l][cl];
        out[c] = t;
    }
}

}  // namespace aether
