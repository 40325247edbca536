// Shared host-side plumbing of the library: error reporting, the device status word that
// bounded waits report into, the launch counter, and the internal entry points of each .cu file.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <atomic>

#include "../../include/aether_b200.h"
#include "launch.cuh"

namespace aether {

// Return codes of every extern "C" entry point (0 = success).
enum : int {
    AE_OK = 0,
    AE_BAD_ARG = -1,       // null pointer, misaligned pointer, non-positive size, workspace too small
    AE_UNSUPPORTED = -2,   // shape/mode the library has no kernel for
    AE_CUDA = -3,          // a CUDA runtime/driver call failed
    AE_DEVICE_TIMEOUT = -4 // an earlier kernel gave up a bounded wait (see aether_device_status)
};

int set_error(int code, const char* fmt, ...);
void count_launch(int n = 1);
// Pinned, device-visible int that kernels write a DeviceStatus code into; allocated once per process.
int* device_status_word();
// Checks cudaGetLastError after a launch; returns AE_OK or AE_CUDA (with message).
int check_launch(const char* what);

// Optional per-kernel timing (off by default): CUDA events recorded around selected launches on the
// launch stream, read back through aether_profile_read.
enum ProfKind : int { PK_IGEMM_FWD = 0, PK_IGEMM_DX = 1, PK_DW = 2, PK_SHADOW = 3, PK_COUNT = 4 };
void prof_begin(int kind, cudaStream_t st);
void prof_end(int kind, cudaStream_t st);

// ---- per-device state.  Kernel attributes (the opt-in to more than 48 KB of dynamic shared memory) and the SM
// count belong to a device, not to the process: a host that drives several GPUs from one process, or switches
// device between calls, gets each of them configured on first use.  The flags are atomics, so any number of host
// threads may call into the library (a doubled cudaFuncSetAttribute is harmless).
static constexpr int AE_MAX_DEVICES = 64;
static inline int current_device() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= AE_MAX_DEVICES) dev = 0;
    return dev;
}
struct PerDeviceSmem {
    std::atomic<int> bytes[AE_MAX_DEVICES];      // largest dynamic shared-memory size configured so far (0: none)
};
// Makes sure `kernel` may be launched with `bytes` of dynamic shared memory on the current device.
template <typename K>
static inline int ensure_dynamic_smem(K kernel, int bytes, PerDeviceSmem& once, const char* what) {
    const int dev = current_device();
    if (once.bytes[dev].load(std::memory_order_acquire) >= bytes) return AE_OK;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return set_error(AE_CUDA, "cudaFuncSetAttribute(%s, %d): %s", what, bytes, cudaGetErrorString(e));
    once.bytes[dev].store(bytes, std::memory_order_release);
    return AE_OK;
}

static inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }
static inline int ceil_div(int a, int b) { return (a + b - 1) / b; }
static inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// ---- conv_simt.cu : fp32 CUDA-core convolution for any filter/stride/padding/channel count, tiled implicit GEMMs
// (`ws`: scratch, nullable; without it tiles that do not fill the SMs are not split)
int simt_conv_fwd(const AetherConvDesc& d, const float* x, const float* w, const float* b, float* y, void* ws, size_t ws_bytes, cudaStream_t st);
int simt_conv_bwd_data(const AetherConvDesc& d, const float* dy, const float* w, float* dx, void* ws, size_t ws_bytes, cudaStream_t st);
int simt_conv_bwd_filter(const AetherConvDesc& d, const float* x, const float* dy, float* dw, float* db, void* ws,
                         size_t ws_bytes, cudaStream_t st);
size_t simt_conv_workspace_bytes(const AetherConvDesc& d);

// ---- conv_split.cu : fp32 convolution on the tensor cores, operands as sums of three bf16 numbers (strides up to 4, any
// channel counts from 16); which shapes gain from it: split_conv_eligible
bool split_conv_eligible(const AetherConvDesc& d);
size_t split_conv_workspace_bytes(const AetherConvDesc& d);
size_t split_conv_fwd_workspace_bytes(const AetherConvDesc& d);      // of that, what a forward pass uses
int split_conv_fwd(const AetherConvDesc& d, const float* x, const float* w, const float* b, float* y, void* ws, cudaStream_t st);
int split_conv_bwd(const AetherConvDesc& d, const float* x, const float* dy, const float* w, float* dx, float* dw, float* db, void* ws,
                   int copies_valid, cudaStream_t st);

// ---- conv_dx_few.cu : dX of first layers (1..4 input channels) on the CUDA cores
int dx_few_conv_bwd_data(const AetherConvDesc& d, const float* dy, const float* w, float* dx, cudaStream_t st);

// ---- conv_generic.cu : classifier heads on the CUDA cores; everything else goes to conv_dx_few.cu and conv_simt.cu
// classifier heads (pointwise, few outputs) with the softmax / the combined softmax and cross-entropy gradient in the kernel
bool generic_head_shape(const AetherConvDesc& d);
int generic_head_softmax_fwd(const AetherConvDesc& d, const float* x, const float* w, const float* b, float* y, float* prob, cudaStream_t st);
int generic_head_bwd(const AetherConvDesc& d, const float* x, const float* dy, const float* w, float* dx, float* dw, float* db, void* ws,
                     size_t ws_bytes, cudaStream_t st);
int generic_head_cce_bwd(const AetherConvDesc& d, const float* prob, const int* labels, const long long* labels64, const float* targets,
                         float smooth, const float* x, const float* w, float* dz, float* dx, float* dw, float* db, void* ws, size_t ws_bytes,
                         cudaStream_t st);
int generic_conv_fwd(const AetherConvDesc& d, const float* x, const float* w, const float* b, float* y, void* ws, size_t ws_bytes,
                     cudaStream_t st);
int generic_conv_bwd_data(const AetherConvDesc& d, const float* dy, const float* w, float* dx, void* ws, size_t ws_bytes, cudaStream_t st);
size_t generic_conv_workspace_bytes(const AetherConvDesc& d);

// ---- conv_smallc.cu : fp32 first-layer convolution (1..4 input channels, fH*fW*Cin <= 64): forward, dW, dB
bool smallc_conv_eligible(const AetherConvDesc& d);
size_t smallc_conv_workspace_bytes(const AetherConvDesc& d);
int smallc_conv_fwd(const AetherConvDesc& d, const float* x, const float* w, const float* b, float* y, float* stats,
                    cudaStream_t st);
long long smallc_conv_stats_blocks(const AetherConvDesc& d);
int smallc_conv_bwd_filter(const AetherConvDesc& d, const float* x, const float* dy, float* dw, float* db, void* ws,
                           size_t ws_bytes, cudaStream_t st);

// ---- conv_first_fp32.cu : the same layers with 3x3 and 5x5 filters, pieces of rows through registers
bool first_fp32_fwd_eligible(const AetherConvDesc& d);
bool first_fp32_dw_eligible(const AetherConvDesc& d);
bool first_fp32_dw_faster(const AetherConvDesc& d);       // than first_tc_bwd_filter without a copy of dy
size_t first_fp32_dw_workspace_bytes(const AetherConvDesc& d);
int first_fp32_fwd(const AetherConvDesc& d, const float* x, const float* w, const float* b, float* y, cudaStream_t st);
int first_fp32_bwd_filter(const AetherConvDesc& d, const float* x, const float* dy, float* dw, float* db, void* ws, size_t ws_bytes, cudaStream_t st);

// The layers behind a convolution that its kernels may apply in inference (pool_epilogue.cuh): Batch_Norm, (leaky) ReLU, 2x2 max pooling.
struct PoolEpilogue {
    const float *gamma, *beta, *mean, *var;
    float eps, alpha;
    float* pooled;
    void* copy;          // nullable: bf16, rows of ld
    int ld;
};

// ---- conv_first_tc.cu : first-layer forward on tensor cores (bf16 mode, thread-built im2col operand)
bool first_tc_eligible(const AetherConvDesc& d);
long long first_tc_stats_blocks(const AetherConvDesc& d);
int first_tc_fwd(const AetherConvDesc& d, const float* x, const float* w, const float* b, float* y, float* stats,
                 cudaStream_t st, const PoolEpilogue* pool = nullptr);
bool first_tc_bwd_eligible(const AetherConvDesc& d);
int first_tc_bwd_filter(const AetherConvDesc& d, const float* x, const float* dy, float* dw, float* db, void* ws,
                        size_t ws_bytes, int dy_colsum_rows, cudaStream_t st);
size_t first_tc_bwd_workspace_bytes(const AetherConvDesc& d);
bool first_tc_operand_layout(const AetherConvDesc& d, AetherOperandLayout* out);
// out[c] = sum over `rows` rows of part[row][C] in fixed order (conv_tc.cu)
int colsum_finish(const float* part, int rows, int C, float* out, cudaStream_t st);
int smallc_reduce_partials(const float* part, int nb, int K, int Cout, float* dw, float* db, cudaStream_t st, const float* colsum = nullptr,
                           int rows = 0);

// ---- conv_tc.cu : tcgen05 implicit-GEMM convolution (stride 1)
bool tc_conv_eligible(const AetherConvDesc& d);
size_t tc_conv_workspace_bytes(const AetherConvDesc& d);
// `stats` (nullable): per-block (count, mean, M2) of every output channel, tc_conv_stats_blocks(d) blocks of [3][Cout]
// A (leaky) ReLU that the forward kernel may apply in its epilogue: its output and, nullable, the bf16 copy of
// that in rows of `ld`.
struct ActEpilogue {
    float* out;
    float alpha;
    void* copy;
    int ld;
};
int tc_conv_fwd(const AetherConvDesc& d, const float* x, const float* w, const float* b, float* y, float* stats, void* ws,
                size_t ws_bytes, int flags, cudaStream_t st, const ActEpilogue* act = nullptr, bool* act_done = nullptr);
bool tc_conv_pool_eligible(const AetherConvDesc& d);
bool tc_conv_pool_faster(const AetherConvDesc& d);
int tc_conv_fwd_pool(const AetherConvDesc& d, const float* x, const float* w, const float* b, const PoolEpilogue& pool, void* ws, size_t ws_bytes, int flags,
                     cudaStream_t st);
int tc_conv_filter_copies(const AetherConvDesc& d, const float* w, void* ws, size_t ws_bytes, cudaStream_t st);
bool tc_conv_operand_layout(const AetherConvDesc& d, AetherOperandLayout* out);
long long tc_conv_stats_blocks(const AetherConvDesc& d);
int tc_conv_bwd(const AetherConvDesc& d, const float* x, const float* dy, const float* w, float* dx, float* dw,
                float* db, void* ws, size_t ws_bytes, int x_shadow_valid, int dy_colsum_rows, cudaStream_t st);

// ---- layers.cu : pieces of Batch_Norm shared with block_fused.cu
int bn_partial_blocks(long long rows);
// (count, mean, M2) partials of x into part, in at most `most` rows; returns their number
int bn_reduce_partials(const float* x, long long rows, int C, float* part, int most, cudaStream_t st);
float* bn_forward_coeffs(const float* x, const float* partials, long long nblocks, const float* gamma, const float* beta,
                         float* running_mean, float* running_var, float* batch_mean, float* batch_var, long long rows,
                         int C, float eps, float momentum, const float* channel_scale, float* ws, cudaStream_t st);
float* bn_eval_coeffs(const float* gamma, const float* beta, const float* running_mean, const float* running_var, int C,
                      float eps, float* ws, cudaStream_t st);
void bn_backward_coeffs(const float* part, int nb, int C, long long rows, const float* gamma, const float* mean,
                        const float* var, float eps, float* dgamma, float* dbeta, float* coeff, const float* pscale,
                        cudaStream_t st);

// a (leaky) ReLU over [rows][C] and the bf16 copy of its output in rows of `ld` (C % 4 == 0, ld % 4 == 0, copy 8-byte aligned)
int act_fwd_copy(const float* x, float* out, float alpha, void* copy, long long rows, int C, int ld, cudaStream_t st);

void bn_backward_apply(const float* x, const float* dy, float* dx, const float* coeff, long long n, int C, cudaStream_t st);

static inline void conv_out_hw(const AetherConvDesc& d, int& Ho, int& Wo) {
    Ho = (d.H + 2 * d.padH - d.fH) / d.sH + 1;
    Wo = (d.W + 2 * d.padW - d.fW) / d.sW + 1;
}

}  // namespace aether
