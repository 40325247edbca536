// The tail of a convolution block of the reference's networks -- Batch_Norm, ReLU / Leaky_ReLU, optional
// Layer_Dropout_Spatial, max Pooling whose windows tile the input (CNN_classes_cupy.py:430-526, 406-428, 384-404,
// 204-312) -- in one pass each way.  The activation between the convolution and the pooling is never written:
//
//   forward : pooled = maxpool( act(x * scale[c] + shift[c]) ), argmax codes kept   (mask folded into scale/shift)
//             reads x once, writes |x|/4 floats + |x|/4 bytes  (layer by layer: 3 reads and 3 writes of |x|)
//   backward: the gradient of an input cell is d_pooled of its window if the cell was the window's maximum, times
//             the activation's derivative, recomputed from x (v = gamma * xhat + beta); a statistics pass and a
//             dx pass, each reading x and d_pooled once.
//
// Every thread owns one window and four channels.  Statistics, running averages, coefficient algebra and the
// fixed-order reductions are the Batch_Norm kernels of layers.cu.
#include <cuda_bf16.h>

#include "common.cuh"
#include "tail.cuh"

namespace aether {

// F > 0: square F x F windows known at compile time -- the window's loads are issued together (one load in flight
// per thread does not cover the HBM latency); F == 0: any window, cells one after the other.
template <int F>
__global__ void __launch_bounds__(256) bn_act_pool_fwd_kernel(const float* __restrict__ x, const float* __restrict__ scale,
                                                              const float* __restrict__ shift, float alpha,
                                                              float* __restrict__ y, uint8_t* __restrict__ arg,
                                                              unsigned total, int W, int C4, int fH_, int fW_, int Wo,
                                                              __nv_bfloat16* __restrict__ copy, int copy_ld,
                                                              float* __restrict__ xsel) {
    pdl_wait();
    const int fH = F ? F : fH_, fW = F ? F : fW_;
    for (unsigned idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
        const unsigned cv = idx % (unsigned)C4;
        unsigned pix = idx / (unsigned)C4;
        const unsigned opix = pix;                             // output pixel of this window
        const unsigned wo = pix % (unsigned)Wo;
        pix /= (unsigned)Wo;                                   // = s * Ho + ho; input rows of all samples are stacked
        const float4 s = *reinterpret_cast<const float4*>(scale + cv * 4);
        const float4 t = *reinterpret_cast<const float4*>(shift + cv * 4);
        const float4* in = reinterpret_cast<const float4*>(x) + ((size_t)pix * fH * W + (size_t)wo * fW) * C4 + cv;
        float4 best = make_float4(0.f, 0.f, 0.f, 0.f), sel = best;     // sel: the input value at the selected cell
        uchar4 code = make_uchar4(0, 0, 0, 0);
        float4 pre[F ? F * F : 1];
        if (F) {
#pragma unroll
            for (int k = 0; k < F * F; ++k) pre[k] = __ldcs(in + ((size_t)(k / (F ? F : 1)) * W + k % (F ? F : 1)) * C4);
        }
#pragma unroll
        for (int i = 0; i < fH; ++i)
#pragma unroll
            for (int j = 0; j < fW; ++j) {
                const float4 v = F ? pre[F ? i * F + j : 0] : __ldcs(in + ((size_t)i * W + j) * C4);
                float4 o;
                o.x = lrelu(fmaf(v.x, s.x, t.x), alpha); o.y = lrelu(fmaf(v.y, s.y, t.y), alpha);
                o.z = lrelu(fmaf(v.z, s.z, t.z), alpha); o.w = lrelu(fmaf(v.w, s.w, t.w), alpha);
                const unsigned char k = (unsigned char)(i * fW + j);
                if (k == 0) {
                    best = o;
                    sel = v;
                } else {                                      // first maximum in row-major window order, as Pooling
                    if (o.x > best.x) { best.x = o.x; code.x = k; sel.x = v.x; }
                    if (o.y > best.y) { best.y = o.y; code.y = k; sel.y = v.y; }
                    if (o.z > best.z) { best.z = o.z; code.z = k; sel.z = v.z; }
                    if (o.w > best.w) { best.w = o.w; code.w = k; sel.w = v.w; }
                }
            }
        if (y != nullptr) reinterpret_cast<float4*>(y)[idx] = best;       // not written when only the bf16 copy is wanted
        reinterpret_cast<uchar4*>(arg)[idx] = code;
        if (copy != nullptr) store_operand_copy(copy, copy_ld, opix, (int)cv, C4, best);
        if (xsel != nullptr) reinterpret_cast<float4*>(xsel)[idx] = sel;
    }
}

// The backward statistics pass when the forward pass kept the input value at every window's selected cell (xsel,
// shaped like the pooled tensor): only that cell has a gradient, so sum(g) and sum(g * xhat) need xsel and d_pooled
// alone -- half of |x| in coalesced reads instead of all of x gathered cell by cell.  part[block][2][C].
__global__ void __launch_bounds__(256) bn_act_pool_bwd_reduce_sel_kernel(
    const float* __restrict__ xsel, const float* __restrict__ dpool, const float* __restrict__ gamma,
    const float* __restrict__ beta, const float* __restrict__ mean, const float* __restrict__ var, float eps, float alpha,
    long long windows, long long win_per_block, int C, float* __restrict__ part) {
    pdl_wait();
    const long long w0 = blockIdx.x * win_per_block;
    long long w1 = w0 + win_per_block;
    if (w1 > windows) w1 = windows;
    const int CV = C >> 2;
    const int cols = CV < 256 ? CV : 256;
    const int lanes = 256 / cols;
    __shared__ float4 sh_a4[256], sh_b4[256];
    for (int cbase = 0; cbase < CV; cbase += cols) {
        const int cv = cbase + threadIdx.x % cols;
        const int rl = threadIdx.x / cols;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
        if (rl < lanes && cv < CV) {
            const int c = cv * 4;
            const float4 mu = *reinterpret_cast<const float4*>(mean + c);
            const float4 vr = *reinterpret_cast<const float4*>(var + c);
            const float4 inv = make_float4(rsqrtf(vr.x + eps), rsqrtf(vr.y + eps), rsqrtf(vr.z + eps), rsqrtf(vr.w + eps));
            const float4 ga = *reinterpret_cast<const float4*>(gamma + c);
            const float4 be = *reinterpret_cast<const float4*>(beta + c);
            const float4* gp = reinterpret_cast<const float4*>(dpool) + cv;
            const float4* xp = reinterpret_cast<const float4*>(xsel) + cv;
#pragma unroll 4
            for (long long wdx = w0 + rl; wdx < w1; wdx += lanes) {
                const float4 g = __ldcs(gp + (size_t)wdx * CV);
                const float4 v = __ldcs(xp + (size_t)wdx * CV);
                const float hx = (v.x - mu.x) * inv.x, hy = (v.y - mu.y) * inv.y;
                const float hz = (v.z - mu.z) * inv.z, hw = (v.w - mu.w) * inv.w;
                const float gx = g.x * lrelu_grad(fmaf(ga.x, hx, be.x), alpha), gy = g.y * lrelu_grad(fmaf(ga.y, hy, be.y), alpha);
                const float gz = g.z * lrelu_grad(fmaf(ga.z, hz, be.z), alpha), gw = g.w * lrelu_grad(fmaf(ga.w, hw, be.w), alpha);
                a.x += gx; a.y += gy; a.z += gz; a.w += gw;
                b.x = fmaf(gx, hx, b.x); b.y = fmaf(gy, hy, b.y); b.z = fmaf(gz, hz, b.z); b.w = fmaf(gw, hw, b.w);
            }
        }
        sh_a4[threadIdx.x] = a;
        sh_b4[threadIdx.x] = b;
        __syncthreads();
        if (threadIdx.x < cols && cv < CV) {
            float* out = part + (size_t)blockIdx.x * 2 * C + cv * 4;
            const float* pa = reinterpret_cast<const float*>(sh_a4);
            const float* pb = reinterpret_cast<const float*>(sh_b4);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                float sa = 0.f, sb = 0.f;
                for (int l = 0; l < lanes; ++l) {
                    sa += pa[(l * cols + threadIdx.x) * 4 + k];
                    sb += pb[(l * cols + threadIdx.x) * 4 + k];
                }
                out[k] = sa;
                out[C + k] = sb;
            }
        }
        __syncthreads();
    }
}

// Per-channel partial sums of g and g * xhat over a slab of windows: part[block][2][C].  Thread = (channel group,
// window lane) like bn_reduce_vec4_kernel; only the window's selected cell has a non-zero g.
__global__ void __launch_bounds__(256) bn_act_pool_bwd_reduce_kernel(
    const float* __restrict__ x, const float* __restrict__ dpool, const uint8_t* __restrict__ arg,
    const float* __restrict__ gamma, const float* __restrict__ beta, const float* __restrict__ mean,
    const float* __restrict__ var, float eps, float alpha, long long windows, long long win_per_block, int W, int C, int fH,
    int fW, int Wo, float* __restrict__ part) {
    pdl_wait();
    const long long w0 = blockIdx.x * win_per_block;
    long long w1 = w0 + win_per_block;
    if (w1 > windows) w1 = windows;
    const int CV = C >> 2;
    const int cols = CV < 256 ? CV : 256;
    const int lanes = 256 / cols;
    __shared__ float4 sh_a4[256], sh_b4[256];
    for (int cbase = 0; cbase < CV; cbase += cols) {
        const int cv = cbase + threadIdx.x % cols;
        const int rl = threadIdx.x / cols;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
        if (rl < lanes && cv < CV) {
            const int c = cv * 4;
            const float4 mu = make_float4(mean[c], mean[c + 1], mean[c + 2], mean[c + 3]);
            const float4 inv = make_float4(rsqrtf(var[c] + eps), rsqrtf(var[c + 1] + eps), rsqrtf(var[c + 2] + eps),
                                           rsqrtf(var[c + 3] + eps));
            const float4 ga = *reinterpret_cast<const float4*>(gamma + c);
            const float4 be = *reinterpret_cast<const float4*>(beta + c);
            for (long long wdx = w0 + rl; wdx < w1; wdx += lanes) {
                const long long pix = wdx / Wo;                // s * Ho + ho
                const int wo = (int)(wdx - pix * Wo);
                const float4 g = (reinterpret_cast<const float4*>(dpool) + cv)[(size_t)wdx * CV];
                const uchar4 cd = (reinterpret_cast<const uchar4*>(arg) + cv)[(size_t)wdx * CV];
                const float4* in = reinterpret_cast<const float4*>(x) + ((size_t)pix * fH * W + (size_t)wo * fW) * CV + cv;
                // the selected cell of each of the four channels (window-local code = i * fW + j)
                const float4 vx = in[((size_t)(cd.x / fW) * W + cd.x % fW) * CV];
                const float4 vy = in[((size_t)(cd.y / fW) * W + cd.y % fW) * CV];
                const float4 vz = in[((size_t)(cd.z / fW) * W + cd.z % fW) * CV];
                const float4 vw = in[((size_t)(cd.w / fW) * W + cd.w % fW) * CV];
                const float hx = (vx.x - mu.x) * inv.x, hy = (vy.y - mu.y) * inv.y;
                const float hz = (vz.z - mu.z) * inv.z, hw = (vw.w - mu.w) * inv.w;
                const float gx = g.x * lrelu_grad(fmaf(ga.x, hx, be.x), alpha), gy = g.y * lrelu_grad(fmaf(ga.y, hy, be.y), alpha);
                const float gz = g.z * lrelu_grad(fmaf(ga.z, hz, be.z), alpha), gw = g.w * lrelu_grad(fmaf(ga.w, hw, be.w), alpha);
                a.x += gx; a.y += gy; a.z += gz; a.w += gw;
                b.x = fmaf(gx, hx, b.x); b.y = fmaf(gy, hy, b.y); b.z = fmaf(gz, hz, b.z); b.w = fmaf(gw, hw, b.w);
            }
        }
        sh_a4[threadIdx.x] = a;
        sh_b4[threadIdx.x] = b;
        __syncthreads();
        if (threadIdx.x < cols && cv < CV) {
            float* out = part + (size_t)blockIdx.x * 2 * C + cv * 4;
            const float* pa = reinterpret_cast<const float*>(sh_a4);
            const float* pb = reinterpret_cast<const float*>(sh_b4);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                float sa = 0.f, sb = 0.f;
                for (int l = 0; l < lanes; ++l) {
                    sa += pa[(l * cols + threadIdx.x) * 4 + k];
                    sb += pb[(l * cols + threadIdx.x) * 4 + k];
                }
                out[k] = sa;
                out[C + k] = sb;
            }
        }
        __syncthreads();
    }
}

// dx = k1 * g + k2 * x + k3 for every cell of every window (g is non-zero only at the window's selected cell).
template <int F>
__global__ void __launch_bounds__(256, 3) bn_act_pool_bwd_apply_kernel(
    const float* __restrict__ x, const float* __restrict__ dpool, const uint8_t* __restrict__ arg,
    const float* __restrict__ gamma, const float* __restrict__ beta, const float* __restrict__ mean,
    const float* __restrict__ var, float eps, float alpha, const float* __restrict__ coeff, float* __restrict__ dx,
    unsigned total, int W, int C, int fH_, int fW_, int Wo, __nv_bfloat16* __restrict__ copy, int copy_ld,
    float* __restrict__ colsum_part) {
    pdl_wait();
    const int fH = F ? F : fH_, fW = F ? F : fW_;
    const int C4 = C >> 2;
    // column sums of dx (the bias gradient of the convolution in front): only with grids whose stride keeps a thread on
    // one channel group (gridDim.x * 256 a multiple of C4; the host checks), so four running sums per thread suffice
    float4 csum = make_float4(0.f, 0.f, 0.f, 0.f);
    // Coefficients of this thread's channels, loaded once where the stride keeps it on them: seven vectors from L1 and four
    // reciprocal roots per window made the L1 the limit (the three block tails of the 128/256/512-channel network
    // at batch 4096: 1440 -> 1230 us).
    const bool fixed = gridDim.x * blockDim.x % (unsigned)C4 == 0;
    float4 k1 = csum, k2 = csum, k3 = csum, mu = csum, ga = csum, be = csum, inv = csum;
    bool loaded = false;
    for (unsigned idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
        const unsigned cv = idx % (unsigned)C4;
        unsigned pix = idx / (unsigned)C4;
        const unsigned wo = pix % (unsigned)Wo;
        pix /= (unsigned)Wo;
        const int c = cv * 4;
        const float4 g = __ldcs(reinterpret_cast<const float4*>(dpool) + idx);
        const uchar4 cd = reinterpret_cast<const uchar4*>(arg)[idx];
        if (!loaded) {
            k1 = *reinterpret_cast<const float4*>(coeff + c);
            k2 = *reinterpret_cast<const float4*>(coeff + C + c);
            k3 = *reinterpret_cast<const float4*>(coeff + 2 * C + c);
            mu = *reinterpret_cast<const float4*>(mean + c);
            ga = *reinterpret_cast<const float4*>(gamma + c);
            be = *reinterpret_cast<const float4*>(beta + c);
            const float4 vr = *reinterpret_cast<const float4*>(var + c);
            inv = make_float4(rsqrtf(vr.x + eps), rsqrtf(vr.y + eps), rsqrtf(vr.z + eps), rsqrtf(vr.w + eps));
            loaded = fixed;
        }
        const size_t first = ((size_t)pix * fH * W + (size_t)wo * fW) * C4 + cv;
        float4 pre[F ? F * F : 1];
        if (F) {
#pragma unroll
            for (int k = 0; k < F * F; ++k)
                pre[k] = __ldcs(reinterpret_cast<const float4*>(x) + first + ((size_t)(k / (F ? F : 1)) * W + k % (F ? F : 1)) * C4);
        }
#pragma unroll
        for (int i = 0; i < fH; ++i)
#pragma unroll
            for (int j = 0; j < fW; ++j) {
                const size_t cell = first + ((size_t)i * W + j) * C4;
                const float4 v = F ? pre[F ? i * F + j : 0] : __ldcs(reinterpret_cast<const float4*>(x) + cell);
                const unsigned char k = (unsigned char)(i * fW + j);
                float4 o;
                o.x = fmaf(k2.x, v.x, k3.x); o.y = fmaf(k2.y, v.y, k3.y); o.z = fmaf(k2.z, v.z, k3.z); o.w = fmaf(k2.w, v.w, k3.w);
                if (cd.x == k) o.x = fmaf(k1.x, g.x * lrelu_grad(fmaf(ga.x, (v.x - mu.x) * inv.x, be.x), alpha), o.x);
                if (cd.y == k) o.y = fmaf(k1.y, g.y * lrelu_grad(fmaf(ga.y, (v.y - mu.y) * inv.y, be.y), alpha), o.y);
                if (cd.z == k) o.z = fmaf(k1.z, g.z * lrelu_grad(fmaf(ga.z, (v.z - mu.z) * inv.z, be.z), alpha), o.z);
                if (cd.w == k) o.w = fmaf(k1.w, g.w * lrelu_grad(fmaf(ga.w, (v.w - mu.w) * inv.w, be.w), alpha), o.w);
                if (dx != nullptr) reinterpret_cast<float4*>(dx)[cell] = o;   // not written when only the bf16 copy is wanted
                if (copy != nullptr) {
                    store_operand_copy(copy, copy_ld, (size_t)pix * fH * W + (size_t)wo * fW + (size_t)i * W + j, (int)cv, C4, o);
                    csum.x += o.x; csum.y += o.y; csum.z += o.z; csum.w += o.w;
                }
            }
    }
    if (colsum_part != nullptr) {
        // threads t, t + C4, ... of the block hold the same four channels: added in that order, one row per block
        __shared__ float4 red[256];
        red[threadIdx.x] = csum;
        __syncthreads();
        if ((int)threadIdx.x < C4) {
            float4 t = red[threadIdx.x];
            for (int l = threadIdx.x + C4; l < 256; l += C4) { const float4 v = red[l]; t.x += v.x; t.y += v.y; t.z += v.z; t.w += v.w; }
            *reinterpret_cast<float4*>(colsum_part + (size_t)blockIdx.x * C + threadIdx.x * 4) = t;
        }
    }
}

// ====================================================================================== block tail, every layer's output kept
// The same chain for a model whose layers each keep their own output (no fusion asked for): Batch_Norm, activation,
// optional spatial dropout, optional max pooling in one pass, writing the output of EVERY layer from registers.  Layer by
// layer the chain reads what the layer before has just written: 4 reads and 3.3 writes of |x| forward against 1 read here,
// 6 reads and 4 writes backward against 3 reads; bound by HBM / L2 bandwidth on large tensors, by launches on small ones
// (five and six launches become one or two and three).
//   forward : bn = x * scale + shift;  act = lrelu(bn);  drop = act * mask (a copy in inference);  pooled, arg
// A thread owns one window (1x1 without pooling) and four channels; cells no window covers (H, W no multiples of the
// window) belong to ragged windows that are not pooled.
template <int F>
__global__ void __launch_bounds__(256) chain_fwd_kernel(const float* __restrict__ x, const float* __restrict__ scale,
                                                        const float* __restrict__ shift, const float* __restrict__ gamma,
                                                        const float* __restrict__ beta, const float* __restrict__ rmean,
                                                        const float* __restrict__ rvar, float eps, float alpha,
                                                        const float* __restrict__ mask, float* __restrict__ bn,
                                                        float* __restrict__ act, float* __restrict__ drop,
                                                        float* __restrict__ pooled, uint8_t* __restrict__ arg, unsigned total, int H,
                                                        int W, int C4, int fH_, int fW_, int Hc, int Wc,
                                                        __nv_bfloat16* __restrict__ copy, int copy_ld) {
    pdl_wait();
    const int fH = F ? F : fH_, fW = F ? F : fW_;
    const int Ho = H / fH, Wo = W / fW;
    // A thread keeps its channels where C / 4 divides the grid's threads (C a power of two): their coefficients are made when the
    // channels change only (inference makes them with a square root and a division per channel, which took as long as the pass's
    // loads: 896 x 32x32x32 pooled 40.6 -> 37 us).
    float4 s, t, k4;
    unsigned cv_now = ~0u;
    for (unsigned idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
        // From the end: what the convolution in front wrote last is still in L2 (37 -> 34 us on 117 MB).
        const unsigned at = total - 1 - idx, cv = at % (unsigned)C4;
        unsigned pix = at / (unsigned)C4;
        const int wo = (int)(pix % (unsigned)Wc);
        pix /= (unsigned)Wc;
        const int ho = (int)(pix % (unsigned)Hc);
        const unsigned smp = pix / (unsigned)Hc;
        if (cv != cv_now) {
            cv_now = cv;
            if (scale != nullptr) {
                s = *reinterpret_cast<const float4*>(scale + cv * 4);
                t = *reinterpret_cast<const float4*>(shift + cv * 4);
            } else {                                          // inference: the coefficients of bn_eval_coeff_kernel
                const float4 g = *reinterpret_cast<const float4*>(gamma + cv * 4), b = *reinterpret_cast<const float4*>(beta + cv * 4);
                const float4 m = *reinterpret_cast<const float4*>(rmean + cv * 4), v = *reinterpret_cast<const float4*>(rvar + cv * 4);
                s = make_float4(g.x / sqrtf(v.x + eps), g.y / sqrtf(v.y + eps), g.z / sqrtf(v.z + eps), g.w / sqrtf(v.w + eps));
                t = make_float4(b.x - m.x * s.x, b.y - m.y * s.y, b.z - m.z * s.z, b.w - m.w * s.w);
            }
            k4 = mask != nullptr ? *reinterpret_cast<const float4*>(mask + cv * 4) : make_float4(1.f, 1.f, 1.f, 1.f);
        }
        const size_t first = (((size_t)smp * H + (size_t)ho * fH) * W + (size_t)wo * fW) * C4 + cv;
        const bool whole = ho < Ho && wo < Wo;                // a ragged window covers cells outside the image, too
        float4 pre[F ? F * F : 1];
        if (F) {
#pragma unroll
            for (int k = 0; k < F * F; ++k)
                if (whole || (ho * F + k / (F ? F : 1) < H && wo * F + k % (F ? F : 1) < W))
                    pre[k] = reinterpret_cast<const float4*>(x)[first + ((size_t)(k / (F ? F : 1)) * W + k % (F ? F : 1)) * C4];
        }
        float4 best = make_float4(0.f, 0.f, 0.f, 0.f);
        uchar4 code = make_uchar4(0, 0, 0, 0);
#pragma unroll
        for (int i = 0; i < fH; ++i)
#pragma unroll
            for (int j = 0; j < fW; ++j) {
                if (!whole && (ho * fH + i >= H || wo * fW + j >= W)) continue;
                const size_t cell = first + ((size_t)i * W + j) * C4;
                const float4 v = F ? pre[F ? i * F + j : 0] : reinterpret_cast<const float4*>(x)[cell];
                float4 o = make_float4(fmaf(v.x, s.x, t.x), fmaf(v.y, s.y, t.y), fmaf(v.z, s.z, t.z), fmaf(v.w, s.w, t.w));
                if (bn != nullptr) reinterpret_cast<float4*>(bn)[cell] = o;
                o = make_float4(lrelu(o.x, alpha), lrelu(o.y, alpha), lrelu(o.z, alpha), lrelu(o.w, alpha));
                if (act != nullptr) reinterpret_cast<float4*>(act)[cell] = o;
                if (drop != nullptr) {
                    if (mask != nullptr) o = make_float4(o.x * k4.x, o.y * k4.y, o.z * k4.z, o.w * k4.w);
                    reinterpret_cast<float4*>(drop)[cell] = o;
                }
                const unsigned char k = (unsigned char)(i * fW + j);
                if (k == 0) {
                    best = o;
                } else {                                      // first maximum in row-major window order, as Pooling
                    if (o.x > best.x) { best.x = o.x; code.x = k; }
                    if (o.y > best.y) { best.y = o.y; code.y = k; }
                    if (o.z > best.z) { best.z = o.z; code.z = k; }
                    if (o.w > best.w) { best.w = o.w; code.w = k; }
                }
            }
        if (pooled != nullptr && whole) {
            const size_t opix = ((size_t)smp * Ho + ho) * Wo + wo;
            reinterpret_cast<float4*>(pooled)[opix * C4 + cv] = best;
            if (arg != nullptr) reinterpret_cast<uchar4*>(arg)[opix * C4 + cv] = code;
            if (copy != nullptr) store_operand_copy(copy, copy_ld, opix, (int)cv, C4, best);
        } else if (pooled == nullptr && copy != nullptr) {
            store_operand_copy(copy, copy_ld, ((size_t)smp * H + ho) * W + wo, (int)cv, C4, best);
        }
    }
}

//   backward: the gradients of every layer's input, and Batch_Norm's sums over the activation's
//     pool_dx = dy at the selected cell;  drop_dx = pool_dx * mask;  act_dx = drop_dx * act'(bn);  sum act_dx, sum act_dx * xhat
// bn = x * scale + shift is recomputed (the same fma, so the same sign as the stored tensor).  Thread = (channel group,
// window lane) over a slab of windows, partials [block][2][C] as in the other statistics passes.
template <int F>
__global__ void __launch_bounds__(256) chain_bwd_kernel(const float* __restrict__ x, const float* __restrict__ dy,
                                                        const uint8_t* __restrict__ arg, const float* __restrict__ scale,
                                                        const float* __restrict__ shift, const float* __restrict__ mean,
                                                        const float* __restrict__ var, float eps, float alpha,
                                                        const float* __restrict__ mask, float* __restrict__ pool_dx,
                                                        float* __restrict__ drop_dx, float* __restrict__ act_dx,
                                                        long long windows, long long win_per_block, int H, int W, int C, int fH_,
                                                        int fW_, int Hc, int Wc, float* __restrict__ part) {
    pdl_wait();
    const int fH = F ? F : fH_, fW = F ? F : fW_;
    const int Ho = H / fH, Wo = W / fW;
    const long long w0 = blockIdx.x * win_per_block;
    long long w1 = w0 + win_per_block;
    if (w1 > windows) w1 = windows;
    const int CV = C >> 2;
    const int cols = CV < 256 ? CV : 256;
    const int lanes = 256 / cols;
    __shared__ float4 sh_a4[256], sh_b4[256];
    for (int cbase = 0; cbase < CV; cbase += cols) {
        const int cv = cbase + threadIdx.x % cols;
        const int rl = threadIdx.x / cols;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
        if (rl < lanes && cv < CV) {
            const int c = cv * 4;
            const float4 mu = make_float4(mean[c], mean[c + 1], mean[c + 2], mean[c + 3]);
            const float4 inv = make_float4(rsqrtf(var[c] + eps), rsqrtf(var[c + 1] + eps), rsqrtf(var[c + 2] + eps),
                                           rsqrtf(var[c + 3] + eps));
            const float4 s = *reinterpret_cast<const float4*>(scale + c), t = *reinterpret_cast<const float4*>(shift + c);
            const float4 k4 = mask != nullptr ? *reinterpret_cast<const float4*>(mask + c) : make_float4(1.f, 1.f, 1.f, 1.f);
            for (long long wdx = w0 + rl; wdx < w1; wdx += lanes) {
                unsigned pix = (unsigned)wdx;
                const int wo = (int)(pix % (unsigned)Wc);
                pix /= (unsigned)Wc;
                const int ho = (int)(pix % (unsigned)Hc);
                const unsigned smp = pix / (unsigned)Hc;
                const bool whole = ho < Ho && wo < Wo;
                const size_t first = (((size_t)smp * H + (size_t)ho * fH) * W + (size_t)wo * fW) * CV + cv;
                float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
                uchar4 cd = make_uchar4(0, 0, 0, 0);
                if (arg == nullptr) {
                    g = reinterpret_cast<const float4*>(dy)[first];
                } else if (whole) {
                    const size_t o = (((size_t)smp * Ho + ho) * Wo + wo) * CV + cv;
                    g = reinterpret_cast<const float4*>(dy)[o];
                    cd = reinterpret_cast<const uchar4*>(arg)[o];
                }
                float4 pre[F ? F * F : 1];
                if (F) {
#pragma unroll
                    for (int k = 0; k < F * F; ++k)
                        if (whole || (ho * F + k / (F ? F : 1) < H && wo * F + k % (F ? F : 1) < W))
                            pre[k] = reinterpret_cast<const float4*>(x)[first + ((size_t)(k / (F ? F : 1)) * W + k % (F ? F : 1)) * CV];
                }
#pragma unroll
                for (int i = 0; i < fH; ++i)
#pragma unroll
                    for (int j = 0; j < fW; ++j) {
                        if (!whole && (ho * fH + i >= H || wo * fW + j >= W)) continue;
                        const size_t cell = first + ((size_t)i * W + j) * CV;
                        const float4 v = F ? pre[F ? i * F + j : 0] : reinterpret_cast<const float4*>(x)[cell];
                        const unsigned char k = (unsigned char)(i * fW + j);
                        float4 d = make_float4(cd.x == k ? g.x : 0.f, cd.y == k ? g.y : 0.f, cd.z == k ? g.z : 0.f, cd.w == k ? g.w : 0.f);
                        if (pool_dx != nullptr) reinterpret_cast<float4*>(pool_dx)[cell] = d;
                        if (drop_dx != nullptr) {
                            d = make_float4(d.x * k4.x, d.y * k4.y, d.z * k4.z, d.w * k4.w);
                            reinterpret_cast<float4*>(drop_dx)[cell] = d;
                        }
                        d.x = fmaf(v.x, s.x, t.x) < 0.f ? alpha * d.x : d.x; d.y = fmaf(v.y, s.y, t.y) < 0.f ? alpha * d.y : d.y;
                        d.z = fmaf(v.z, s.z, t.z) < 0.f ? alpha * d.z : d.z; d.w = fmaf(v.w, s.w, t.w) < 0.f ? alpha * d.w : d.w;
                        reinterpret_cast<float4*>(act_dx)[cell] = d;
                        a.x += d.x; a.y += d.y; a.z += d.z; a.w += d.w;
                        b.x = fmaf(d.x, (v.x - mu.x) * inv.x, b.x); b.y = fmaf(d.y, (v.y - mu.y) * inv.y, b.y);
                        b.z = fmaf(d.z, (v.z - mu.z) * inv.z, b.z); b.w = fmaf(d.w, (v.w - mu.w) * inv.w, b.w);
                    }
            }
        }
        sh_a4[threadIdx.x] = a;
        sh_b4[threadIdx.x] = b;
        __syncthreads();
        if (threadIdx.x < cols && cv < CV) {
            float* out = part + (size_t)blockIdx.x * 2 * C + cv * 4;
            const float* pa = reinterpret_cast<const float*>(sh_a4);
            const float* pb = reinterpret_cast<const float*>(sh_b4);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                float sa = 0.f, sb = 0.f;
                for (int l = 0; l < lanes; ++l) {
                    sa += pa[(l * cols + threadIdx.x) * 4 + k];
                    sb += pb[(l * cols + threadIdx.x) * 4 + k];
                }
                out[k] = sa;
                out[C + k] = sb;
            }
        }
        __syncthreads();
    }
}

// dx = k1 * g + k2 * x + k3, with the bf16 operand copy of dx and its column sums for the convolution in front
// (C / 4 divides 256: a thread keeps its four channels).
__global__ void __launch_bounds__(256) chain_apply_copy_kernel(const float* __restrict__ x, const float* __restrict__ g_,
                                                               const float* __restrict__ coeff, float* __restrict__ dx, long long n4,
                                                               int C, __nv_bfloat16* __restrict__ copy, int copy_ld,
                                                               float* __restrict__ colsum_part) {
    pdl_wait();
    const int C4 = C >> 2;
    const int cv = threadIdx.x % C4, c = cv * 4;
    const float4 k1 = *reinterpret_cast<const float4*>(coeff + c);
    const float4 k2 = *reinterpret_cast<const float4*>(coeff + C + c);
    const float4 k3 = *reinterpret_cast<const float4*>(coeff + 2 * C + c);
    float4 csum = make_float4(0.f, 0.f, 0.f, 0.f);
    const long long stride = (long long)gridDim.x * 256;
#pragma unroll 2
    for (long long i = blockIdx.x * 256LL + threadIdx.x; i < n4; i += stride) {
        const float4 v = reinterpret_cast<const float4*>(x)[i];
        const float4 g = reinterpret_cast<const float4*>(g_)[i];
        float4 o;
        o.x = fmaf(k1.x, g.x, fmaf(k2.x, v.x, k3.x));
        o.y = fmaf(k1.y, g.y, fmaf(k2.y, v.y, k3.y));
        o.z = fmaf(k1.z, g.z, fmaf(k2.z, v.z, k3.z));
        o.w = fmaf(k1.w, g.w, fmaf(k2.w, v.w, k3.w));
        reinterpret_cast<float4*>(dx)[i] = o;
        store_operand_copy(copy, copy_ld, (size_t)((unsigned long long)i / (unsigned)C4), cv, C4, o);
        csum.x += o.x; csum.y += o.y; csum.z += o.z; csum.w += o.w;
    }
    __shared__ float4 red[256];
    red[threadIdx.x] = csum;
    __syncthreads();
    if ((int)threadIdx.x < C4) {
        float4 t = red[threadIdx.x];
        for (int l = threadIdx.x + C4; l < 256; l += C4) { const float4 v = red[l]; t.x += v.x; t.y += v.y; t.z += v.z; t.w += v.w; }
        *reinterpret_cast<float4*>(colsum_part + (size_t)blockIdx.x * C + threadIdx.x * 4) = t;
    }
}

static int fused_blocks(long long items, int threads, int per_sm) {
    long long b = (items + threads - 1) / threads;
    const long long cap = 148LL * per_sm;
    if (b > cap) b = cap;
    return (int)(b < 1 ? 1 : b);
}

static int block_check(const char* who, int S, int H, int W, int C, int fH, int fW, float alpha, long long* windows4) {
    if (S <= 0 || H <= 0 || W <= 0 || C <= 0 || fH <= 0 || fW <= 0) return set_error(AE_BAD_ARG, "%s: non-positive dimension", who);
    if (C % 4 || H % fH || W % fW || fH * fW > 255)
        return set_error(AE_UNSUPPORTED, "%s: needs C %% 4 == 0 and pooling windows that tile the input (H=%d W=%d f=%dx%d C=%d)",
                         who, H, W, fH, fW, C);
    if (!(alpha >= 0.f && alpha < 1.f)) return set_error(AE_BAD_ARG, "%s: alpha must be in [0, 1)", who);
    *windows4 = 1LL * S * (H / fH) * (W / fW) * (C / 4);
    if (*windows4 >= (1LL << 32) - (1LL << 22)) return set_error(AE_UNSUPPORTED, "%s: tensor too large for 32-bit window indices", who);
    return AE_OK;
}

}  // namespace aether

using namespace aether;

extern "C" size_t aether_bn_workspace_bytes(int64_t rows, int C);

extern "C" int aether_bn_act_pool_fwd(const float* x, const float* partials, int64_t nblocks, const float* gamma,
                                      const float* beta, float* running_mean, float* running_var, float* batch_mean,
                                      float* batch_var, float* pooled, uint8_t* argmax, int S, int H, int W, int C, int fH,
                                      int fW, float eps, float momentum, float alpha, const float* channel_scale,
                                      int training, void* ws, size_t ws_bytes, void* stream) {
    return aether_bn_act_pool_fwd_copy(x, partials, nblocks, gamma, beta, running_mean, running_var, batch_mean, batch_var,
                                       pooled, argmax, S, H, W, C, fH, fW, eps, momentum, alpha, channel_scale, training,
                                       nullptr, 0, nullptr, ws, ws_bytes, stream);
}

extern "C" int aether_bn_act_pool_fwd_copy(const float* x, const float* partials, int64_t nblocks, const float* gamma,
                                           const float* beta, float* running_mean, float* running_var, float* batch_mean,
                                           float* batch_var, float* pooled, uint8_t* argmax, int S, int H, int W, int C,
                                           int fH, int fW, float eps, float momentum, float alpha,
                                           const float* channel_scale, int training, void* operand_copy, int copy_ld,
                                           float* selected_x, void* ws, size_t ws_bytes, void* stream) {
    if (!x || !gamma || !beta || !running_mean || !running_var || (!pooled && !operand_copy) || !argmax || !ws ||
        (training && (!batch_mean || !batch_var)))
        return set_error(AE_BAD_ARG, "aether_bn_act_pool_fwd: null pointer");
    if (operand_copy && (copy_ld < C || copy_ld % 4 || (reinterpret_cast<uintptr_t>(operand_copy) & 7)))
        return set_error(AE_BAD_ARG, "aether_bn_act_pool_fwd_copy: operand copy needs ld >= C, ld %% 4 == 0, 8-byte alignment");
    if (selected_x && !aligned16(selected_x)) return set_error(AE_BAD_ARG, "aether_bn_act_pool_fwd_copy: selected_x must be 16-byte aligned");
    long long windows4 = 0;
    int rc = block_check("aether_bn_act_pool_fwd", S, H, W, C, fH, fW, alpha, &windows4);
    if (rc) return rc;
    if (!aligned16(x) || (pooled && !aligned16(pooled)) || !aligned16(ws) || (reinterpret_cast<uintptr_t>(argmax) & 3))
        return set_error(AE_BAD_ARG, "aether_bn_act_pool_fwd: arrays must be 16-byte aligned (argmax: 4)");
    const long long rows = 1LL * S * H * W;
    if (ws_bytes < aether_bn_workspace_bytes(rows, C)) return set_error(AE_BAD_ARG, "aether_bn_act_pool_fwd: workspace too small");
    if (partials && (nblocks <= 0 || nblocks > (1 << 30))) return set_error(AE_BAD_ARG, "aether_bn_act_pool_fwd: nblocks");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (training && bn_small(rows, C)) {
        BnSmallFwd p = {};
        p.x = x;
        p.part = partials;
        p.nblocks = (int)nblocks;
        if (!partials) {
            p.part = static_cast<float*>(ws);
            p.nblocks = bn_reduce_partials(x, rows, C, static_cast<float*>(ws), 148, st);
        }
        p.gamma = gamma; p.beta = beta; p.running_mean = running_mean; p.running_var = running_var;
        p.batch_mean = batch_mean; p.batch_var = batch_var; p.eps = eps; p.momentum = momentum; p.alpha = alpha;
        p.mask = channel_scale;
        p.fold = 1;
        p.pooled = pooled; p.arg = argmax; p.xsel = selected_x; p.copy = static_cast<__nv_bfloat16*>(operand_copy); p.copy_ld = copy_ld;
        p.H = H; p.W = W; p.C = C; p.fH = fH; p.fW = fW; p.Hc = H / fH; p.Wc = W / fW;
        p.windows = (unsigned)(windows4 / (C / 4));
        bn_small_forward(p, st);
        return check_launch("aether_bn_act_pool_fwd");
    }
    float* coeff = training ? bn_forward_coeffs(x, partials, nblocks, gamma, beta, running_mean, running_var, batch_mean,
                                                batch_var, rows, C, eps, momentum, channel_scale, static_cast<float*>(ws), st)
                            : bn_eval_coeffs(gamma, beta, running_mean, running_var, C, eps, static_cast<float*>(ws), st);
    const int fb = fused_blocks(windows4, 256, 16);
    __nv_bfloat16* copy = static_cast<__nv_bfloat16*>(operand_copy);
    if (fH == 2 && fW == 2)
        launch(bn_act_pool_fwd_kernel<2>, fb, 256, 0, st, x, coeff, coeff + C, alpha, pooled, argmax, (unsigned)windows4, W, C / 4, fH, fW,
               W / fW, copy, copy_ld, selected_x);
    else
        launch(bn_act_pool_fwd_kernel<0>, fb, 256, 0, st, x, coeff, coeff + C, alpha, pooled, argmax, (unsigned)windows4, W, C / 4, fH, fW,
               W / fW, copy, copy_ld, selected_x);
    count_launch();
    return check_launch("aether_bn_act_pool_fwd");
}

extern "C" int aether_bn_act_pool_bwd(const float* x, const float* dpooled, const uint8_t* argmax, const float* gamma,
                                      const float* beta, const float* batch_mean, const float* batch_var, float* dx,
                                      float* dgamma, float* dbeta, int S, int H, int W, int C, int fH, int fW, float eps,
                                      float alpha, const float* channel_scale, void* ws, size_t ws_bytes, void* stream) {
    return aether_bn_act_pool_bwd_copy(x, dpooled, argmax, gamma, beta, batch_mean, batch_var, dx, dgamma, dbeta, S, H, W, C, fH,
                                       fW, eps, alpha, channel_scale, nullptr, 0, nullptr, 0, nullptr, nullptr, ws, ws_bytes, stream);
}

extern "C" int aether_bn_act_pool_bwd_copy(const float* x, const float* dpooled, const uint8_t* argmax, const float* gamma,
                                           const float* beta, const float* batch_mean, const float* batch_var, float* dx,
                                           float* dgamma, float* dbeta, int S, int H, int W, int C, int fH, int fW, float eps,
                                           float alpha, const float* channel_scale, void* operand_copy, int copy_ld,
                                           float* colsum_part, int colsum_rows_max, int* colsum_rows,
                                           const float* selected_x, void* ws, size_t ws_bytes, void* stream) {
    if (!x || !dpooled || !argmax || !gamma || !beta || !batch_mean || !batch_var || (!dx && !operand_copy) || !dgamma ||
        !dbeta || !ws)
        return set_error(AE_BAD_ARG, "aether_bn_act_pool_bwd: null pointer");
    if (operand_copy) {
        if (copy_ld < C || copy_ld % 4 || (reinterpret_cast<uintptr_t>(operand_copy) & 7) || !colsum_part || !colsum_rows ||
            colsum_rows_max < 1 || !aligned16(colsum_part))
            return set_error(AE_BAD_ARG, "aether_bn_act_pool_bwd_copy: operand copy needs ld >= C, ld %% 4 == 0, 8-byte alignment "
                                         "and a column-sum buffer");
        if (256 % (C / 4 > 0 ? C / 4 : 1) || C / 4 > 256)
            return set_error(AE_UNSUPPORTED, "aether_bn_act_pool_bwd_copy: the column sums need C / 4 to divide 256 (C = %d)", C);
    }
    long long windows4 = 0;
    int rc = block_check("aether_bn_act_pool_bwd", S, H, W, C, fH, fW, alpha, &windows4);
    if (rc) return rc;
    if (!aligned16(x) || !aligned16(dpooled) || (dx && !aligned16(dx)) || !aligned16(ws) || !aligned16(gamma) || !aligned16(beta) ||
        !aligned16(batch_mean) || !aligned16(batch_var) || (reinterpret_cast<uintptr_t>(argmax) & 3))
        return set_error(AE_BAD_ARG, "aether_bn_act_pool_bwd: arrays must be 16-byte aligned (argmax: 4)");
    const long long rows = 1LL * S * H * W;
    if (ws_bytes < aether_bn_workspace_bytes(rows, C)) return set_error(AE_BAD_ARG, "aether_bn_act_pool_bwd: workspace too small");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const long long windows = windows4 / (C / 4);
    const bool small = bn_small(rows, C);
    int nb = bn_partial_blocks(rows);
    if (nb > windows) nb = (int)windows;
    if (small && nb > 148) nb = 148;
    float* part = static_cast<float*>(ws);
    float* coeff = part + (size_t)bn_partial_blocks(rows) * 3 * C;
    if (selected_x) {
        if (!aligned16(selected_x)) return set_error(AE_BAD_ARG, "aether_bn_act_pool_bwd_copy: selected_x must be 16-byte aligned");
        launch(bn_act_pool_bwd_reduce_sel_kernel, nb, 256, 0, st, selected_x, dpooled, gamma, beta, batch_mean, batch_var, eps, alpha,
               windows, (windows + nb - 1) / nb, C, part);
    } else {
        launch(bn_act_pool_bwd_reduce_kernel, nb, 256, 0, st, x, dpooled, argmax, gamma, beta, batch_mean, batch_var, eps, alpha, windows,
               (windows + nb - 1) / nb, W, C, fH, fW, W / fW, part);
    }
    count_launch();
    if (small) {
        BnSmallBwd p = {};
        p.x = x; p.dy = dpooled; p.arg = argmax; p.part = part; p.nblocks = nb; p.gamma = gamma; p.beta = beta; p.mean = batch_mean;
        p.var = batch_var; p.pscale = channel_scale; p.eps = eps; p.alpha = alpha; p.dgamma = dgamma; p.dbeta = dbeta; p.dx = dx;
        p.copy = static_cast<__nv_bfloat16*>(operand_copy); p.copy_ld = copy_ld; p.colsum_part = operand_copy ? colsum_part : nullptr;
        p.W = W; p.C = C; p.fH = fH; p.fW = fW;
        p.windows = (unsigned)windows;
        p.rows = rows;
        const int sums = bn_small_backward(p, operand_copy ? colsum_rows_max : 0, st);
        if (operand_copy) *colsum_rows = sums;
        return check_launch("aether_bn_act_pool_bwd");
    }
    bn_backward_coeffs(part, nb, C, rows, gamma, batch_mean, batch_var, eps, dgamma, dbeta, coeff, channel_scale, st);
    int fb = fused_blocks(windows4, 256, 3);     // what is resident at once: equal shares, coefficients loaded once per thread
    __nv_bfloat16* copy = static_cast<__nv_bfloat16*>(operand_copy);
    if (copy) {                                  // one row of column sums per CTA: no more CTAs than rows offered
        if (fb > colsum_rows_max) fb = colsum_rows_max;
        *colsum_rows = fb;
    }
    if (fH == 2 && fW == 2)
        launch(bn_act_pool_bwd_apply_kernel<2>, fb, 256, 0, st, x, dpooled, argmax, gamma, beta, batch_mean, batch_var, eps, alpha, coeff,
               dx, (unsigned)windows4, W, C, fH, fW, W / fW, copy, copy_ld, copy ? colsum_part : nullptr);
    else
        launch(bn_act_pool_bwd_apply_kernel<0>, fb, 256, 0, st, x, dpooled, argmax, gamma, beta, batch_mean, batch_var, eps, alpha, coeff,
               dx, (unsigned)windows4, W, C, fH, fW, W / fW, copy, copy_ld, copy ? colsum_part : nullptr);
    count_launch();
    return check_launch("aether_bn_act_pool_bwd");
}

extern "C" int aether_chain_fwd(const float* x, const float* partials, int64_t nblocks, const float* gamma, const float* beta,
                                float* running_mean, float* running_var, float* batch_mean, float* batch_var, float* bn_out,
                                float* act_out, float* drop_out, float* pooled, uint8_t* argmax, int S, int H, int W, int C, int fH,
                                int fW, float eps, float momentum, float alpha, const float* mask, int training, void* operand_copy,
                                int copy_ld, void* ws, size_t ws_bytes, void* stream) {
    if (!x || !gamma || !beta || !running_mean || !running_var || !ws || (mask && !drop_out) ||
        (training ? (!batch_mean || !batch_var || !bn_out || !act_out || (pooled && !argmax)) : (!act_out && !drop_out && !pooled)))
        return set_error(AE_BAD_ARG, "aether_chain_fwd: null pointer");
    if (S <= 0 || H <= 0 || W <= 0 || C <= 0 || fH <= 0 || fW <= 0 || (!pooled && (fH != 1 || fW != 1)))
        return set_error(AE_BAD_ARG, "aether_chain_fwd: bad dimension");
    if (!(alpha >= 0.f && alpha < 1.f)) return set_error(AE_BAD_ARG, "aether_chain_fwd: alpha must be in [0, 1)");
    const long long items = 1LL * S * ceil_div(H, fH) * ceil_div(W, fW) * (C / 4);
    if (C % 4 || fH * fW > 255 || items >= (1LL << 32) - (1LL << 22))
        return set_error(AE_UNSUPPORTED, "aether_chain_fwd: needs C %% 4 == 0, windows of at most 255 cells, 32-bit window indices");
    if (!aligned16(x) || (bn_out && !aligned16(bn_out)) || (act_out && !aligned16(act_out)) || (drop_out && !aligned16(drop_out)) ||
        (pooled && !aligned16(pooled)) || !aligned16(gamma) || !aligned16(beta) || !aligned16(running_mean) || !aligned16(running_var) || (mask && !aligned16(mask)) || !aligned16(ws) ||
        (argmax && (reinterpret_cast<uintptr_t>(argmax) & 3)))
        return set_error(AE_BAD_ARG, "aether_chain_fwd: arrays must be 16-byte aligned (argmax: 4)");
    if (operand_copy && (copy_ld < C || copy_ld % 4 || (reinterpret_cast<uintptr_t>(operand_copy) & 7)))
        return set_error(AE_BAD_ARG, "aether_chain_fwd: operand copy needs ld >= C, ld %% 4 == 0, 8-byte alignment");
    const long long rows = 1LL * S * H * W;
    if (ws_bytes < aether_bn_workspace_bytes(rows, C)) return set_error(AE_BAD_ARG, "aether_chain_fwd: workspace too small");
    if (partials && (nblocks <= 0 || nblocks > (1 << 30))) return set_error(AE_BAD_ARG, "aether_chain_fwd: nblocks");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (training && bn_small(rows, C, BN_SMALL_CHAIN)) {
        BnSmallFwd p = {};
        p.x = x;
        p.part = partials;
        p.nblocks = (int)nblocks;
        if (!partials) {
            p.part = static_cast<float*>(ws);
            p.nblocks = bn_reduce_partials(x, rows, C, static_cast<float*>(ws), 148, st);
        }
        p.gamma = gamma; p.beta = beta; p.running_mean = running_mean; p.running_var = running_var;
        p.batch_mean = batch_mean; p.batch_var = batch_var; p.eps = eps; p.momentum = momentum; p.alpha = alpha; p.mask = mask;
        p.coeff = static_cast<float*>(ws) + (size_t)bn_partial_blocks(rows) * 3 * C;
        p.bn_out = bn_out; p.act_out = act_out; p.drop_out = drop_out; p.pooled = pooled; p.arg = argmax;
        p.copy = static_cast<__nv_bfloat16*>(operand_copy); p.copy_ld = copy_ld;
        p.H = H; p.W = W; p.C = C; p.fH = fH; p.fW = fW; p.Hc = ceil_div(H, fH); p.Wc = ceil_div(W, fW);
        p.windows = (unsigned)(items / (C / 4));
        bn_small_forward(p, st);
        return check_launch("aether_chain_fwd");
    }
    const float* coeff = nullptr;
    if (training)
        coeff = bn_forward_coeffs(x, partials, nblocks, gamma, beta, running_mean, running_var, batch_mean, batch_var, rows, C, eps,
                                  momentum, nullptr, static_cast<float*>(ws), st);
    const float* shift = coeff ? coeff + C : nullptr;
    const int fb = fused_blocks(items, 256, 16);
    const auto kernel = fH == 2 && fW == 2 ? chain_fwd_kernel<2> : fH == 1 && fW == 1 ? chain_fwd_kernel<1> : chain_fwd_kernel<0>;
    launch(kernel, fb, 256, 0, st, x, coeff, shift, gamma, beta, running_mean, running_var, eps, alpha, mask, bn_out, act_out, drop_out,
           pooled, argmax, (unsigned)items, H, W, C / 4, fH, fW, ceil_div(H, fH), ceil_div(W, fW), static_cast<__nv_bfloat16*>(operand_copy),
           copy_ld);
    count_launch();
    return check_launch("aether_chain_fwd");
}

extern "C" int aether_chain_bwd(const float* x, const float* dy, const uint8_t* argmax, const float* gamma, const float* batch_mean,
                                const float* batch_var, float* pool_dx, float* drop_dx, float* act_dx, float* dx, float* dgamma,
                                float* dbeta, int S, int H, int W, int C, int fH, int fW, float eps, float alpha, const float* mask,
                                void* operand_copy, int copy_ld, float* colsum_part, int colsum_rows_max, int* colsum_rows, void* ws,
                                size_t ws_bytes, void* stream) {
    if (!x || !dy || !gamma || !batch_mean || !batch_var || !act_dx || !dx || !dgamma || !dbeta || !ws || (argmax && !pool_dx) ||
        (mask && !drop_dx))
        return set_error(AE_BAD_ARG, "aether_chain_bwd: null pointer");
    if (S <= 0 || H <= 0 || W <= 0 || C <= 0 || fH <= 0 || fW <= 0 || (!argmax && (fH != 1 || fW != 1)))
        return set_error(AE_BAD_ARG, "aether_chain_bwd: bad dimension");
    if (!(alpha >= 0.f && alpha < 1.f)) return set_error(AE_BAD_ARG, "aether_chain_bwd: alpha must be in [0, 1)");
    const long long windows = 1LL * S * ceil_div(H, fH) * ceil_div(W, fW);
    if (C % 4 || fH * fW > 255 || windows >= (1LL << 32))
        return set_error(AE_UNSUPPORTED, "aether_chain_bwd: needs C %% 4 == 0, windows of at most 255 cells, 32-bit window indices");
    if (!aligned16(x) || !aligned16(dy) || !aligned16(act_dx) || !aligned16(dx) || (pool_dx && !aligned16(pool_dx)) ||
        (drop_dx && !aligned16(drop_dx)) || (mask && !aligned16(mask)) || !aligned16(ws) || (argmax && (reinterpret_cast<uintptr_t>(argmax) & 3)))
        return set_error(AE_BAD_ARG, "aether_chain_bwd: arrays must be 16-byte aligned (argmax: 4)");
    if (operand_copy) {
        if (copy_ld < C || copy_ld % 4 || (reinterpret_cast<uintptr_t>(operand_copy) & 7) || !colsum_part || !colsum_rows ||
            colsum_rows_max < 1 || !aligned16(colsum_part))
            return set_error(AE_BAD_ARG, "aether_chain_bwd: operand copy needs ld >= C, ld %% 4 == 0, 8-byte alignment and a column-sum buffer");
        if (C / 4 > 256 || 256 % (C / 4)) return set_error(AE_UNSUPPORTED, "aether_chain_bwd: the column sums need C / 4 to divide 256 (C = %d)", C);
    }
    const long long rows = 1LL * S * H * W;
    if (ws_bytes < aether_bn_workspace_bytes(rows, C)) return set_error(AE_BAD_ARG, "aether_chain_bwd: workspace too small");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    float* part = static_cast<float*>(ws);
    float* coeff = part + (size_t)bn_partial_blocks(rows) * 3 * C;        // still the forward pass's scale and shift
    const bool small = bn_small(rows, C, BN_SMALL_CHAIN);
    int nb = bn_partial_blocks(rows);
    if (nb > windows) nb = (int)windows;
    if (small && nb > 148 * 2) nb = 148 * 2;
    const auto kernel = fH == 2 && fW == 2 ? chain_bwd_kernel<2> : fH == 1 && fW == 1 ? chain_bwd_kernel<1> : chain_bwd_kernel<0>;
    launch(kernel, nb, 256, 0, st, x, dy, argmax, coeff, coeff + C, batch_mean, batch_var, eps, alpha, mask, pool_dx, drop_dx, act_dx, windows,
           (windows + nb - 1) / nb, H, W, C, fH, fW, ceil_div(H, fH), ceil_div(W, fW), part);
    count_launch();
    if (small) {
        BnSmallBwd p = {};
        p.x = x; p.dy = act_dx; p.part = part; p.nblocks = nb; p.gamma = gamma; p.mean = batch_mean; p.var = batch_var; p.eps = eps;
        p.alpha = -1.f; p.dgamma = dgamma; p.dbeta = dbeta; p.dx = dx; p.copy = static_cast<__nv_bfloat16*>(operand_copy); p.copy_ld = copy_ld;
        p.colsum_part = operand_copy ? colsum_part : nullptr;
        p.W = p.fH = p.fW = 1; p.C = C;
        p.windows = (unsigned)rows;
        p.rows = rows;
        const int sums = bn_small_backward(p, operand_copy ? colsum_rows_max : 0, st);
        if (operand_copy) *colsum_rows = sums;
        return check_launch("aether_chain_bwd");
    }
    bn_backward_coeffs(part, nb, C, rows, gamma, batch_mean, batch_var, eps, dgamma, dbeta, coeff, nullptr, st);
    const long long n4 = rows * (C / 4);
    if (operand_copy) {
        int fb = fused_blocks(n4, 256, 8);
        if (fb > colsum_rows_max) fb = colsum_rows_max;
        *colsum_rows = fb;
        launch(chain_apply_copy_kernel, fb, 256, 0, st, x, act_dx, coeff, dx, n4, C, static_cast<__nv_bfloat16*>(operand_copy), copy_ld,
               colsum_part);
        count_launch();
    } else {
        bn_backward_apply(x, act_dx, dx, coeff, rows * C, C, st);
    }
    return check_launch("aether_chain_bwd");
}
