// Stores of accumulator blocks by the filter-gradient kernels.
#pragma once
#include <stddef.h>
#include <stdint.h>

namespace aether {

// A 32x32 block (lane = row, v[k] = column k: the shape tcgen05.ld leaves it in) into a row-major fp32 matrix, limited to
// `rows` and `cols` (a multiple of 4) of it.  Stored from the registers, an instruction would write 16 bytes of 32 rows;
// through 36-float rows of shared memory (no bank conflicts either way) it writes four whole 128-byte lines.
static constexpr int STORE_BLOCK_FLOATS = 32 * 36;

__device__ __forceinline__ void store_block_32x32(float* stage, const uint32_t (&v)[32], float* dst, size_t ld, int rows, int cols,
                                                  int lane) {
#pragma unroll
    for (int c4 = 0; c4 < 8; ++c4)
        *reinterpret_cast<uint4*>(stage + lane * 36 + 4 * c4) = make_uint4(v[4 * c4], v[4 * c4 + 1], v[4 * c4 + 2], v[4 * c4 + 3]);
    __syncwarp();
    const int c = (lane & 7) * 4;
    if (c < cols) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = i * 4 + (lane >> 3);
            if (r < rows) *reinterpret_cast<float4*>(dst + (size_t)r * ld + c) = *reinterpret_cast<const float4*>(stage + r * 36 + c);
        }
    }
    __syncwarp();
}

}  // namespace aether
