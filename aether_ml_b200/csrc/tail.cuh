// What the block-tail kernels (Batch_Norm + activation + dropout + pooling) share.
#pragma once
#include <cuda_bf16.h>

#include "common.cuh"

namespace aether {

// Operand copy hand-off.  The tensor these passes write (the pooled activation going forward, dx going back) is the
// next convolution's x, respectively the previous convolution's dy, whose tensor-core kernels read a bf16 copy with
// the channels padded to `ld`.  When the consumer's workspace is known the copy is written here, from the values
// already in registers, instead of by a cast pass that reads the fp32 tensor again: 4 channels = 8 bytes per thread,
// and the threads of the first channel groups also zero the padding [C, ld) of their pixel.
__device__ __forceinline__ void store_operand_copy(__nv_bfloat16* copy, int ld, size_t pixel, int cv, int C4, float4 v) {
    __nv_bfloat162 o[2] = {__floats2bfloat162_rn(v.x, v.y), __floats2bfloat162_rn(v.z, v.w)};
    __nv_bfloat16* row = copy + pixel * (size_t)ld;
    *reinterpret_cast<uint2*>(row + cv * 4) = *reinterpret_cast<uint2*>(o);
    for (int pg = C4 + cv; pg * 4 < ld; pg += C4) *reinterpret_cast<uint2*>(row + pg * 4) = make_uint2(0u, 0u);
}
__device__ __forceinline__ float lrelu(float v, float alpha) { return v > 0.f ? v : alpha * v; }
// derivative of the activation at pre-activation v (the reference passes the gradient at v == 0, :412-428)
__device__ __forceinline__ float lrelu_grad(float v, float alpha) { return v < 0.f ? alpha : 1.f; }

// ---- bn_small.cu: one-pass forms for small tensors.  A CTA works on 32 channels, so what counts is the rows times the channels
// filled up to whole blocks of 32.  Measured on B200, one-pass against three-launch form in us, forward + backward:
//   Batch_Norm alone, with the activation or with pooling: 1M x 4 (32M filled) 59 + 36 / 27 + 17, 128K x 8 (4M) 18 + 10 / 18 + 10,
//     512K x 8 (16M) 34 + 23 / 21 + 16, 128K x 16 (4M) 16 + 11 / 15 + 12, 128K x 32 (4M) 15 + 13 / 16 + 16, 192K x 32 (6M) 19 + 23 /
//     18 + 20, 32K x 256 (8M) 26 + 31 / 23 + 29;
//   every layer's output kept (the pass writes four times as much): 128K x 32 (4M) 18 + 22 / 19 + 25, 192K x 32 (6M) 26 + 33 / 25 + 35,
//     256K x 32 (8M) 36 + 43 / 31 + 46, 256K x 8 (8M) 24 + 21 / 19 + 21.
static constexpr long long BN_SMALL = 4LL << 20, BN_SMALL_CHAIN = 7LL << 20;

struct BnSmallFwd {
    const float* x;
    const float* part;            // [nblocks][3][C] (count, mean, M2)
    int nblocks;
    const float *gamma, *beta;
    float *running_mean, *running_var, *batch_mean, *batch_var;
    float* coeff;                 // nullable: scale and shift, 2 * C floats (without the mask)
    float eps, momentum, alpha;   // alpha < 0: no activation
    const float* mask;            // nullable: channel factors of a spatial dropout
    int fold;                     // the mask multiplies scale and shift instead of the activation
    float *bn_out, *act_out, *drop_out, *pooled, *xsel;      // each nullable
    uint8_t* arg;
    __nv_bfloat16* copy;
    int copy_ld;
    int H, W, C, fH, fW, Hc, Wc;  // windows of the input, ragged ones included: Hc x Wc per sample
    unsigned windows;
};
struct BnSmallBwd {
    const float *x, *dy;          // dy: per window (1x1 windows: per cell)
    const uint8_t* arg;           // nullable: selected cell of each window
    const float* part;            // [nblocks][2][C]
    int nblocks;
    const float *gamma, *beta, *mean, *var, *pscale;
    float eps, alpha;             // alpha < 0: dy is not taken through an activation
    float *dgamma, *dbeta, *dx;   // dx nullable with copy
    __nv_bfloat16* copy;
    int copy_ld;
    float* colsum_part;           // with copy: one row per chunk
    int W, C, fH, fW;
    unsigned windows;
    long long rows;
};
bool bn_small(long long rows, int C, long long most = BN_SMALL);
void bn_small_forward(const BnSmallFwd& p, cudaStream_t st);
// Returns the rows of column sums written (at most rows_max, when that is positive).
int bn_small_backward(const BnSmallBwd& p, int rows_max, cudaStream_t st);

}  // namespace aether
