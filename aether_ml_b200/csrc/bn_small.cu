// Batch_Norm (and the activation, spatial dropout and pooling behind it) on tensors that fit in L2: the merge of the
// statistics partials runs inside the pass over the data instead of in a launch of its own.
//
// A small tensor's pass takes three to five microseconds, and the finalize kernels before it (layers.cu) five to seven: a
// handful of CTAs on a chain of L2 round trips.  Here the grid is channel blocks of 32 x chunks of the pixels, one CTA of 32
// warps per SM; every CTA merges the partials of its own 32 channels (the producers write at most two rows of partials per
// CTA, 296: 114 KB out of L2 per CTA, which is why there is one per SM and not two; double precision, fixed order -- the same
// bits in every CTA), and the coefficients go straight from shared memory into its pass.  The first chunk's CTA writes the
// statistics.  (Clusters of four CTAs that share the merge through distributed shared memory start later than they save.)
// What a thread reads first of its windows is on its way while the merge runs (forward pass of 128 x 32x32x32, 16x16x64, 8x8x128: 10.7, 9.0, 7.8 -> 10.5, 8.8,
// 7.5 us); going back the activation's derivative is taken at the selected cell only and its coefficients come out of shared memory, so that 64
// registers hold a window (13.7, 10.9, 8.4 -> 12.6, 9.2, 7.5 us; of 376 bytes of spills 64 are left, around the merge).
// Only below BN_SMALL (tail.cuh): a large tensor is a stream of HBM traffic, for which the CTAs' 128-byte pieces and the
// repeated merge cost more than the 7 us they save.
#include <cuda_bf16.h>

#include "common.cuh"
#include "sm100_ptx.cuh"
#include "stats_epilogue.cuh"
#include "tail.cuh"
#include "tc_host.cuh"

namespace aether {

static constexpr int BNS_THREADS = 1024, BNS_WARPS = BNS_THREADS / 32, BNS_LANES = BNS_THREADS / 8;

// Sums of NQ quantities over the partial rows for the 32 channels of this CTA: out[q][channel] in shared memory.
// f(entries, values[NQ]) turns the NQ entries of one partial row into what is summed.
template <int NQ, typename F>
__device__ __forceinline__ void merge_partials(double (*red)[BNS_WARPS][32], const float* __restrict__ part, int nblocks, int C, int c,
                                               bool c_ok, F f) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int U = 5;                                 // rows in flight per warp (296 rows: two round trips to L2)
    double s[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) s[q] = 0.0;
    if (c_ok)
        for (int b = warp; b < nblocks; b += U * BNS_WARPS) {
            float t[U][NQ];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int q = 0; q < NQ; ++q)
                    t[u][q] = b + u * BNS_WARPS < nblocks ? part[((size_t)(b + u * BNS_WARPS) * NQ + q) * C + c] : 0.f;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                double v[NQ];
                f(t[u], v);
#pragma unroll
                for (int q = 0; q < NQ; ++q) s[q] += v[q];
            }
        }
#pragma unroll
    for (int q = 0; q < NQ; ++q) red[q][warp][lane] = s[q];
    __syncthreads();
    if (warp < NQ) {                                     // one warp per quantity adds the warps' sums, in order
        double t[4] = {0.0, 0.0, 0.0, 0.0};              // (four chains: a double add takes long)
#pragma unroll
        for (int w = 0; w < BNS_WARPS; ++w) t[w & 3] += red[warp][w][lane];
        red[warp][0][lane] = (t[0] + t[1]) + (t[2] + t[3]);
    }
    __syncthreads();
}

template <int F>
__global__ void __launch_bounds__(BNS_THREADS, 1) bn_small_fwd_kernel(const BnSmallFwd p) {
    pdl_wait();
    __shared__ double red[3][BNS_WARPS][32];
    __shared__ __align__(16) float sc_s[32], sh_s[32], mk_s[32];
    const int ncb = (p.C + 31) >> 5;
    const int cb = blockIdx.x % ncb, chunk = blockIdx.x / ncb, chunks = gridDim.x / ncb;
    const int g8 = threadIdx.x & 7, C4 = p.C >> 2, cv = cb * 8 + g8;
    const int fH = F ? F : p.fH, fW = F ? F : p.fW;
    const int Ho = p.H / fH, Wo = p.W / fW;
    // a thread's next window: its first value and, of windows of a known size, all of them
    unsigned win = chunk * BNS_LANES + (threadIdx.x >> 3), smp = 0;
    int ho = 0, wo = 0;
    unsigned first = 0;                                  // (32 bits: BN_SMALL)
    bool whole = false;
    float4 pre[F ? F * F : 1];
    auto load = [&]() {
        if (win >= p.windows || cv >= C4) return;
        wo = (int)(win % (unsigned)p.Wc);
        const unsigned r = win / (unsigned)p.Wc;
        ho = (int)(r % (unsigned)p.Hc);
        smp = r / (unsigned)p.Hc;
        first = ((smp * p.H + ho * fH) * p.W + wo * fW) * C4 + cv;
        whole = ho < Ho && wo < Wo;
        if (F) {
#pragma unroll
            for (int k = 0; k < F * F; ++k)
                if (whole || (ho * F + k / (F ? F : 1) < p.H && wo * F + k % (F ? F : 1) < p.W))
                    pre[k] = reinterpret_cast<const float4*>(p.x)[first + ((unsigned)(k / (F ? F : 1)) * p.W + k % (F ? F : 1)) * C4];
        }
    };
    load();                                              // (does not wait for the merge)
    {
        const int c = cb * 32 + (threadIdx.x & 31);
        float ga = 0.f, be = 0.f, mk = 1.f;
        if (threadIdx.x < 32 && c < p.C) {
            ga = p.gamma[c];
            be = p.beta[c];
            if (p.mask != nullptr) mk = p.mask[c];
        }
        merge_partials<3>(red, p.part, p.nblocks, p.C, c, c < p.C, [](const float (&q)[3], double (&v)[3]) {
            stats_row_terms(q[0], q[1], q[2], v[0], v[1], v[2]);
        });
        if (threadIdx.x < 32) {                          // as bn_finalize_fwd_kernel
            float sc = 0.f, sh = 0.f;
            if (c < p.C) {
                const double N = red[0][0][threadIdx.x], S1 = red[1][0][threadIdx.x], Q = red[2][0][threadIdx.x];
                const double rN = N > 0 ? 1.0 / N : 0.0, M = S1 * rN;
                double M2 = Q - N * M * M;
                if (M2 < 0.0) M2 = 0.0;
                const double var = M2 * rN;
                const double s = (double)ga * rsqrt(var + (double)p.eps);
                sc = (float)s;
                sh = (float)((double)be - M * s);
                if (chunk == 0) {
                    p.batch_mean[c] = (float)M;
                    p.batch_var[c] = (float)var;
                    p.running_mean[c] = p.momentum * p.running_mean[c] + (1.f - p.momentum) * (float)M;
                    p.running_var[c] = p.momentum * p.running_var[c] + (1.f - p.momentum) * (float)var;
                    if (p.coeff != nullptr) {
                        p.coeff[c] = sc;
                        p.coeff[p.C + c] = sh;
                    }
                }
                if (p.fold) { sc *= mk; sh *= mk; }      // act(v) * m = act(m * v), m >= 0
            }
            sc_s[threadIdx.x] = sc;
            sh_s[threadIdx.x] = sh;
            mk_s[threadIdx.x] = mk;
        }
        __syncthreads();
    }
    if (cv >= C4) return;
    const float4 s = *reinterpret_cast<const float4*>(sc_s + 4 * g8), t = *reinterpret_cast<const float4*>(sh_s + 4 * g8);
    const float4 k4 = *reinterpret_cast<const float4*>(mk_s + 4 * g8);
    const bool act = p.alpha >= 0.f;
    for (; win < p.windows; win += chunks * BNS_LANES, load()) {
        float4 best = make_float4(0.f, 0.f, 0.f, 0.f), sel = best;
        uchar4 code = make_uchar4(0, 0, 0, 0);
#pragma unroll
        for (int i = 0; i < fH; ++i)
#pragma unroll
            for (int j = 0; j < fW; ++j) {
                if (!whole && (ho * fH + i >= p.H || wo * fW + j >= p.W)) continue;
                const unsigned cell = first + ((unsigned)i * p.W + j) * C4;
                const float4 v = F ? pre[F ? i * F + j : 0] : reinterpret_cast<const float4*>(p.x)[cell];
                float4 o = make_float4(fmaf(v.x, s.x, t.x), fmaf(v.y, s.y, t.y), fmaf(v.z, s.z, t.z), fmaf(v.w, s.w, t.w));
                if (p.bn_out != nullptr) reinterpret_cast<float4*>(p.bn_out)[cell] = o;
                if (act) o = make_float4(lrelu(o.x, p.alpha), lrelu(o.y, p.alpha), lrelu(o.z, p.alpha), lrelu(o.w, p.alpha));
                if (p.act_out != nullptr) reinterpret_cast<float4*>(p.act_out)[cell] = o;
                if (p.drop_out != nullptr) {
                    o = make_float4(o.x * k4.x, o.y * k4.y, o.z * k4.z, o.w * k4.w);
                    reinterpret_cast<float4*>(p.drop_out)[cell] = o;
                }
                const unsigned char k = (unsigned char)(i * fW + j);
                if (k == 0) {
                    best = o;
                    sel = v;
                } else {                                  // first maximum in row-major window order, as Pooling
                    if (o.x > best.x) { best.x = o.x; code.x = k; sel.x = v.x; }
                    if (o.y > best.y) { best.y = o.y; code.y = k; sel.y = v.y; }
                    if (o.z > best.z) { best.z = o.z; code.z = k; sel.z = v.z; }
                    if (o.w > best.w) { best.w = o.w; code.w = k; sel.w = v.w; }
                }
            }
        if (!whole) continue;
        const unsigned opix = (smp * Ho + ho) * Wo + wo;
        if (p.pooled != nullptr) reinterpret_cast<float4*>(p.pooled)[opix * C4 + cv] = best;
        if (p.arg != nullptr) reinterpret_cast<uchar4*>(p.arg)[opix * C4 + cv] = code;
        if (p.xsel != nullptr) reinterpret_cast<float4*>(p.xsel)[opix * C4 + cv] = sel;
        if (p.copy != nullptr) store_operand_copy(p.copy, p.copy_ld, opix, cv, C4, best);
    }
}

// dx = k1 * g + k2 * x + k3 with g = dy [* act'(gamma * xhat + beta)] at every cell, or at the selected cell of each pooling
// window only; the merge is bn_finalize_bwd_kernel's.
template <int F>
__global__ void __launch_bounds__(BNS_THREADS, 1) bn_small_bwd_kernel(const BnSmallBwd p) {
    pdl_wait();
    __shared__ double red[2][BNS_WARPS][32];
    __shared__ __align__(16) float k_s[3][32], act_s[4][32];
    const int ncb = (p.C + 31) >> 5;
    const int cb = blockIdx.x % ncb, chunk = blockIdx.x / ncb, chunks = gridDim.x / ncb;
    const int g8 = threadIdx.x & 7, C4 = p.C >> 2, cv = cb * 8 + g8, c4 = cv * 4;
    const bool c_ok = cv < C4;
    const int fH = F ? F : p.fH, fW = F ? F : p.fW;
    const int Wo = p.W / fW;                              // (pooling windows tile the input here)
    unsigned win = chunk * BNS_LANES + (threadIdx.x >> 3);
    unsigned first = 0;
    float4 g = make_float4(0.f, 0.f, 0.f, 0.f), pre[F ? F * F : 1];
    uchar4 cd = make_uchar4(0, 0, 0, 0);
    auto load = [&]() {
        if (win >= p.windows || !c_ok) return;
        const int wo = (int)(win % (unsigned)Wo);
        const unsigned hrow = win / (unsigned)Wo;         // s * Ho + ho
        first = hrow * fH * p.W + wo * fW;
        g = reinterpret_cast<const float4*>(p.dy)[win * C4 + cv];
        if (p.arg != nullptr) cd = reinterpret_cast<const uchar4*>(p.arg)[win * C4 + cv];
        if (F) {
#pragma unroll
            for (int k = 0; k < F * F; ++k)
                pre[k] = reinterpret_cast<const float4*>(p.x)[(first + (unsigned)(k / (F ? F : 1)) * p.W + k % (F ? F : 1)) * C4 + cv];
        }
    };
    load();                                               // (does not wait for the merge)
    {
        const int c = cb * 32 + (threadIdx.x & 31);
        float ga = 0.f, be = 0.f, va = 0.f, me = 0.f, ps = 1.f;
        if (threadIdx.x < 32 && c < p.C) {
            ga = p.gamma[c];
            va = p.var[c];
            me = p.mean[c];
            if (p.beta != nullptr) be = p.beta[c];
            if (p.pscale != nullptr) ps = p.pscale[c];
        }
        merge_partials<2>(red, p.part, p.nblocks, p.C, c, c < p.C, [](const float (&q)[2], double (&v)[2]) {
            v[0] = q[0];
            v[1] = q[1];
        });
        if (threadIdx.x < 32) {
            float k1 = 0.f, k2 = 0.f, k3 = 0.f;
            if (c < p.C) {
                const double ms = ps;
                const double sdy = red[0][0][threadIdx.x] * ms, sdyx = red[1][0][threadIdx.x] * ms;
                const double inv = rsqrt((double)va + (double)p.eps), rN = 1.0 / (double)p.rows;
                const double g = ga, d2 = -g * inv * inv * sdyx * rN;
                k1 = (float)(g * inv * ms);
                k2 = (float)d2;
                k3 = (float)(-g * inv * sdy * rN - d2 * (double)me);
                if (chunk == 0) {
                    p.dgamma[c] = (float)sdyx;
                    p.dbeta[c] = (float)sdy;
                }
            }
            k_s[0][threadIdx.x] = k1;
            k_s[1][threadIdx.x] = k2;
            k_s[2][threadIdx.x] = k3;
            act_s[0][threadIdx.x] = me;
            act_s[1][threadIdx.x] = rsqrtf(va + p.eps);
            act_s[2][threadIdx.x] = ga;
            act_s[3][threadIdx.x] = be;
        }
        __syncthreads();
    }
    float4 csum = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c_ok) {
        const float4 k1 = *reinterpret_cast<const float4*>(k_s[0] + 4 * g8), k2 = *reinterpret_cast<const float4*>(k_s[1] + 4 * g8);
        const float4 k3 = *reinterpret_cast<const float4*>(k_s[2] + 4 * g8);
        const bool act = p.alpha >= 0.f;
        auto coeffs = [&](int k) {                        // (out of shared memory for every window: sixteen registers fewer)
            float4 v;
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(smem_u32(act_s[k] + 4 * g8)));
            return v;
        };
        // dy of a window's selected cell, whose value is v, through the activation
        auto back = [&](float4 v) {
            if (!act) return g;
            const float4 mu = coeffs(0), inv = coeffs(1), ga = coeffs(2), be = coeffs(3);
            return make_float4(g.x * lrelu_grad(fmaf(ga.x, (v.x - mu.x) * inv.x, be.x), p.alpha), g.y * lrelu_grad(fmaf(ga.y, (v.y - mu.y) * inv.y, be.y), p.alpha),
                               g.z * lrelu_grad(fmaf(ga.z, (v.z - mu.z) * inv.z, be.z), p.alpha), g.w * lrelu_grad(fmaf(ga.w, (v.w - mu.w) * inv.w, be.w), p.alpha));
        };
        for (; win < p.windows; win += chunks * BNS_LANES, load()) {
            float4 d = g;
            if (F) {
                float4 v = pre[0];
#pragma unroll
                for (int k = 1; k < F * F; ++k) {
                    if (cd.x == k) v.x = pre[k].x;
                    if (cd.y == k) v.y = pre[k].y;
                    if (cd.z == k) v.z = pre[k].z;
                    if (cd.w == k) v.w = pre[k].w;
                }
                d = back(v);
            }
#pragma unroll
            for (int i = 0; i < fH; ++i)
#pragma unroll
                for (int j = 0; j < fW; ++j) {
                    const unsigned pixel = first + (unsigned)i * p.W + j, cell = pixel * C4 + cv;
                    const float4 v = F ? pre[F ? i * F + j : 0] : reinterpret_cast<const float4*>(p.x)[cell];
                    const unsigned char k = (unsigned char)(i * fW + j);
                    float4 o = make_float4(fmaf(k2.x, v.x, k3.x), fmaf(k2.y, v.y, k3.y), fmaf(k2.z, v.z, k3.z), fmaf(k2.w, v.w, k3.w));
                    if (!F) d = back(v);
                    if (cd.x == k) o.x = fmaf(k1.x, d.x, o.x);
                    if (cd.y == k) o.y = fmaf(k1.y, d.y, o.y);
                    if (cd.z == k) o.z = fmaf(k1.z, d.z, o.z);
                    if (cd.w == k) o.w = fmaf(k1.w, d.w, o.w);
                    if (p.dx != nullptr) reinterpret_cast<float4*>(p.dx)[cell] = o;
                    if (p.copy != nullptr) {
                        store_operand_copy(p.copy, p.copy_ld, pixel, cv, C4, o);
                        csum.x += o.x; csum.y += o.y; csum.z += o.z; csum.w += o.w;
                    }
                }
        }
    }
    if (p.colsum_part != nullptr) {                       // one row of column sums per chunk; this CTA's 32 columns of it
        float4* sums = reinterpret_cast<float4*>(red);    // the merge's staging, no longer needed
#pragma unroll
        for (int o = 8; o <= 16; o *= 2) {
            csum.x += __shfl_xor_sync(0xffffffffu, csum.x, o); csum.y += __shfl_xor_sync(0xffffffffu, csum.y, o);
            csum.z += __shfl_xor_sync(0xffffffffu, csum.z, o); csum.w += __shfl_xor_sync(0xffffffffu, csum.w, o);
        }
        __syncthreads();
        if ((threadIdx.x & 31) < 8) sums[(threadIdx.x >> 5) * 8 + g8] = csum;
        __syncthreads();
        if (threadIdx.x < 8 && c_ok) {
            float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int l = 0; l < BNS_WARPS; ++l) { const float4 v = sums[l * 8 + threadIdx.x]; t.x += v.x; t.y += v.y; t.z += v.z; t.w += v.w; }
            *reinterpret_cast<float4*>(p.colsum_part + (size_t)chunk * p.C + c4) = t;
        }
    }
}

// CTAs of a pass: one per SM in whole channel blocks, no more chunks than there are rounds of windows.
static int small_chunks(int C, unsigned windows, int most) {
    const int ncb = ceil_div(C, 32);
    int chunks = num_sms() / ncb;
    const int rounds = (int)((windows + BNS_LANES - 1) / BNS_LANES);
    if (chunks > rounds) chunks = rounds;
    if (most > 0 && chunks > most) chunks = most;
    return chunks < 1 ? 1 : chunks;
}

bool bn_small(long long rows, int C, long long most) { return C % 4 == 0 && rows * (ceil_div(C, 32) * 32LL) <= most; }

void bn_small_forward(const BnSmallFwd& p, cudaStream_t st) {
    const int grid = small_chunks(p.C, p.windows, 0) * ceil_div(p.C, 32);
    const auto kernel = p.fH == 2 && p.fW == 2 ? bn_small_fwd_kernel<2> : p.fH == 1 && p.fW == 1 ? bn_small_fwd_kernel<1> : bn_small_fwd_kernel<0>;
    launch(kernel, grid, BNS_THREADS, 0, st, p);
    count_launch();
}

int bn_small_backward(const BnSmallBwd& p, int rows_max, cudaStream_t st) {
    const int chunks = small_chunks(p.C, p.windows, rows_max);
    const auto kernel = p.fH == 2 && p.fW == 2 ? bn_small_bwd_kernel<2> : p.fH == 1 && p.fW == 1 ? bn_small_bwd_kernel<1> : bn_small_bwd_kernel<0>;
    launch(kernel, chunks * ceil_div(p.C, 32), BNS_THREADS, 0, st, p);
    count_launch();
    return chunks;
}

}  // namespace aether
