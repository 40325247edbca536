// What a convolution's epilogue does in inference with the layers behind it: Batch_Norm by its running statistics, (leaky) ReLU and max pooling over
// 2x2 windows, in the arithmetic of the pass over the convolution's output that it takes the place of (chain_fwd_kernel, block_fused.cu).
#pragma once
#include <cuda_bf16.h>

#include "common.cuh"
#include "tail.cuh"

namespace aether {

// Scale and shift of channel c.
__device__ __forceinline__ void pool_coefficients(const PoolEpilogue& e, int c, int C, float& scale, float& shift) {
    scale = shift = 0.f;
    if (c >= C) return;
    scale = e.gamma[c] / sqrtf(e.var[c] + e.eps);
    shift = e.beta[c] - e.mean[c] * scale;
}
__device__ __forceinline__ float4 pool_activation(float4 y, float4 s, float4 t, float alpha) {
    return make_float4(lrelu(fmaf(y.x, s.x, t.x), alpha), lrelu(fmaf(y.y, s.y, t.y), alpha), lrelu(fmaf(y.z, s.z, t.z), alpha), lrelu(fmaf(y.w, s.w, t.w), alpha));
}
// The first maximum in row-major window order, as Pooling (a NaN stays only where it comes first).
__device__ __forceinline__ float4 pool_first_max(float4 a, float4 b, float4 c, float4 d) {
    auto first = [](float p, float q, float r, float s) {
        float m = p;
        if (q > m) m = q;
        if (r > m) m = r;
        return s > m ? s : m;
    };
    return make_float4(first(a.x, b.x, c.x, d.x), first(a.y, b.y, c.y, d.y), first(a.z, b.z, c.z, d.z), first(a.w, b.w, c.w, d.w));
}
// Four channels of window `at`: the pooled values and their operand copy, zero in the columns of padding.
__device__ __forceinline__ void pool_store(const PoolEpilogue& e, long long at, int col, int C, float4 v) {
    if (col < C) *reinterpret_cast<float4*>(e.pooled + at * C + col) = v;
    if (e.copy != nullptr && col < e.ld) {
        const bool in = col < C;
        const __nv_bfloat162 o[2] = {__floats2bfloat162_rn(in ? v.x : 0.f, in ? v.y : 0.f), __floats2bfloat162_rn(in ? v.z : 0.f, in ? v.w : 0.f)};
        *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(e.copy) + at * e.ld + col) = *reinterpret_cast<const uint2*>(o);
    }
}

}  // namespace aether
