// First layers (1..4 input channels, 3x3 and 5x5 filters, columns at stride 1) in single precision: the forward pass and the filter gradient.
//
//   y[p][d] = b[d] + sum_k col[p][k] * w[k][d],   dw[k][d] = sum_p col[p][k] * dy[p][d],   db[d] = sum_p dy[p][d]   (CNN_classes_cupy.py:70-161)
//
// Bound by the FMA pipes where there are three input channels, by the traffic of y and dy with one.  A thread has four output channels and walks a
// piece of an output row; `lanes` threads next to each other have all channels of it.  Filter, respectively gradient, stays in registers over all its
// pieces, and so do the input columns under the filter: a step of one pixel loads one new column, of which every value meets the four channels as
// pairs (fma.rn.f32x2).  A pixel of a 3x3 filter on three channels is 9 loads and 54 FMAs (pairs) of a warp.  Columns and dy are
// loaded F pixels ahead.
// With eight warps of 240 registers an SM the FMA pipes are busy for 45 (forward) and 35 % of the time, the rest goes to latencies that two warps of a scheduler do not
// cover.  Measured, us, against the im2col tiles of conv_smallc.cu and conv_simt.cu, forward and filter gradient with its reduction: 211 x 28x28 3->16
// 16.1 + 45.1 / 9.0 + 13.2, 256 x 64x64 3->32 109 + 200 / 69 + 92, 215 x 33x34 1->32 14.2 + 48.3 / 9.3 + 14.4, 216 x 28x28 3->20 18.4 + 34.0 / 9.6 + 15.0, 100 x
// 40x40 4->64 filter gradient 64 / 41, 313 x 29x24 3->28 5x5 60 / 37.  Windows loaded anew for every pixel, dy through a ring of bulk copies: 114 for the second's
// gradient; prefetching dy into L1 further ahead: slower by a tenth; three input channels by single filter rows: 112.
#include <math.h>
#include <string.h>

#include "common.cuh"
#include "tc_host.cuh"

namespace aether {

static constexpr int FP_THREADS = 256;
__host__ __device__ constexpr int fp_ctas(int values) { return values <= 12 ? 2 : 1; }       // of an SM, by the registers that the values take

struct FirstWalk {
    const float* x;
    int S, H, W, sH, pH, pW, Ho, Wo;
    int Cout, lanes, groups;         // threads of a pixel, pieces that a CTA walks at once
    int segs, T;                     // pieces of a row, pixels of a piece
    int units;                       // pieces
};
__device__ __forceinline__ unsigned long long fp_pair(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void fp_fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long fp_add2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float fp_lo(unsigned long long v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float fp_hi(unsigned long long v) { return __uint_as_float((unsigned)(v >> 32)); }

// A piece of an output row and the input columns under its pixels, filter rows [R0, R0 + RP): column c of the piece is the first of pixel c.
template <int CIN, int F, int R0, int RP>
struct FirstPiece {
    static constexpr int V = RP * CIN;
    const float* row[RP];            // column 0
    bool in[RP];
    int c0, W, len;                  // image column of column 0, pixels
    size_t pixel;                    // of the output
    __device__ __forceinline__ void set(const FirstWalk& g, int unit) {
        const unsigned r = (unsigned)unit / (unsigned)g.segs, n = r / (unsigned)g.Ho;
        const int w0 = (int)(unit - r * g.segs) * g.T, h0 = (int)(r - n * g.Ho) * g.sH - g.pH + R0;
        c0 = w0 - g.pW;
        W = g.W;
        len = min(g.T, g.Wo - w0);
        pixel = (size_t)r * g.Wo + w0;
#pragma unroll
        for (int i = 0; i < RP; ++i) {
            in[i] = (unsigned)(h0 + i) < (unsigned)g.H;
            row[i] = g.x + (((long long)n * g.H + h0 + i) * g.W + c0) * CIN;          // (may lie before the image)
        }
    }
    __device__ __forceinline__ void column(int c, float (&v)[V]) const {
        const bool ok = (unsigned)(c0 + c) < (unsigned)W && c < len + F - 1;
#pragma unroll
        for (int i = 0; i < RP; ++i)
#pragma unroll
            for (int k = 0; k < CIN; ++k) v[i * CIN + k] = ok && in[i] ? __ldg(row[i] + c * CIN + k) : 0.f;
    }
};

// ---------------------------------------------------------------------------------- forward
template <int CIN, int F>
__global__ void __launch_bounds__(FP_THREADS, fp_ctas(CIN * F * F)) first_fp32_fwd_kernel(const FirstWalk g, const float* __restrict__ weights, const float* __restrict__ bias,
                                                                       float* __restrict__ y) {
    constexpr int V = F * CIN;
    pdl_wait();
    const int t = min((int)threadIdx.x, g.groups * g.lanes - 1), grp = t / g.lanes, d0 = (t - grp * g.lanes) * 4;
    const bool idle = (int)threadIdx.x != t, vec = g.Cout % 4 == 0;
    unsigned long long w[F * V][2];
    float b[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) b[c] = bias != nullptr && d0 + c < g.Cout ? bias[d0 + c] : 0.f;
#pragma unroll
    for (int k = 0; k < F * V; ++k) {
        float v[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) v[c] = d0 + c < g.Cout ? weights[k * g.Cout + d0 + c] : 0.f;
        w[k][0] = fp_pair(v[0], v[1]);
        w[k][1] = fp_pair(v[2], v[3]);
    }
    for (int unit = blockIdx.x * g.groups + grp; unit < g.units; unit += gridDim.x * g.groups) {
        FirstPiece<CIN, F, 0, F> piece;
        piece.set(g, unit);
        unsigned long long win[F][V];
        float next[F][V];
#pragma unroll
        for (int u = 0; u < F - 1; ++u) {
            piece.column(u, next[u]);
#pragma unroll
            for (int e = 0; e < V; ++e) win[u][e] = fp_pair(next[u][e], next[u][e]);
        }
#pragma unroll
        for (int u = 0; u < F; ++u) piece.column(F - 1 + u, next[u]);
        float* o = y + piece.pixel * g.Cout + d0;
        for (int k = 0; k < piece.len; k += F)
#pragma unroll
            for (int u = 0; u < F; ++u, o += g.Cout) {
                constexpr int LAST = F - 1;
#pragma unroll
                for (int e = 0; e < V; ++e) win[(u + LAST) % F][e] = fp_pair(next[u][e], next[u][e]);
                piece.column(k + u + F + LAST, next[u]);
                if (k + u >= piece.len) continue;
                unsigned long long acc[F][2];
#pragma unroll
                for (int i = 0; i < F; ++i) acc[i][0] = acc[i][1] = 0ull;
#pragma unroll
                for (int j = 0; j < F; ++j)
#pragma unroll
                    for (int i = 0; i < F; ++i)
#pragma unroll
                        for (int c = 0; c < CIN; ++c)
#pragma unroll
                            for (int h = 0; h < 2; ++h) fp_fma2(acc[i][h], win[(u + j) % F][i * CIN + c], w[(i * F + j) * CIN + c][h]);
#pragma unroll
                for (int i = 1; i < F; ++i)
#pragma unroll
                    for (int h = 0; h < 2; ++h) acc[0][h] = fp_add2(acc[0][h], acc[i][h]);
                const float r[4] = {fp_lo(acc[0][0]) + b[0], fp_hi(acc[0][0]) + b[1], fp_lo(acc[0][1]) + b[2], fp_hi(acc[0][1]) + b[3]};
                if (idle) continue;
                if (vec) {
                    *reinterpret_cast<float4*>(o) = make_float4(r[0], r[1], r[2], r[3]);
                } else {
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (d0 + c < g.Cout) o[c] = r[c];
                }
            }
    }
}

// ---------------------------------------------------------------------------------- filter gradient
// Filters of more than 27 values go by single rows, each with CTAs of its own.  The sums of a CTA's groups meet in shared memory, the CTAs' in
// smallc_reduce_partials, both in fixed order.
__host__ __device__ constexpr int fd_rows(int CIN, int F) { return CIN * F * F <= 27 ? F : 1; }

template <int CIN, int F, int R0>
__device__ __forceinline__ void first_dw_rows(const FirstWalk& g, const float* __restrict__ dy, float* __restrict__ part, int cta, int ctas, float* red) {
    constexpr int RP = fd_rows(CIN, F), V = RP * CIN, KN = F * V, NV = KN + 1, K = CIN * F * F;
    const int t = min((int)threadIdx.x, g.groups * g.lanes - 1), grp = t / g.lanes, d0 = (t - grp * g.lanes) * 4;
    const bool idle = (int)threadIdx.x != t, vec = g.Cout % 4 == 0;
    unsigned long long acc[NV][2];                           // (the last: sums of dy)
#pragma unroll
    for (int k = 0; k < NV; ++k) acc[k][0] = acc[k][1] = 0ull;
    for (int unit = cta * g.groups + grp; unit < g.units; unit += ctas * g.groups) {
        FirstPiece<CIN, F, R0, RP> piece;
        piece.set(g, unit);
        const float* o = dy + piece.pixel * g.Cout + d0;
        auto load = [&](int k) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            const float* s = o + (size_t)k * g.Cout;
            if (k < piece.len) {
                if (vec) {
                    v = __ldg(reinterpret_cast<const float4*>(s));
                } else {
                    v.x = __ldg(s);
                    if (d0 + 1 < g.Cout) v.y = __ldg(s + 1);
                    if (d0 + 2 < g.Cout) v.z = __ldg(s + 2);
                    if (d0 + 3 < g.Cout) v.w = __ldg(s + 3);
                }
            }
            return v;
        };
        unsigned long long win[F][V];
        float next[F][V];
        float4 dyn[F];
#pragma unroll
        for (int u = 0; u < F; ++u) dyn[u] = load(u);
#pragma unroll
        for (int u = 0; u < F - 1; ++u) {
            piece.column(u, next[u]);
#pragma unroll
            for (int e = 0; e < V; ++e) win[u][e] = fp_pair(next[u][e], next[u][e]);
        }
#pragma unroll
        for (int u = 0; u < F; ++u) piece.column(F - 1 + u, next[u]);
        for (int k = 0; k < piece.len; k += F)
#pragma unroll
            for (int u = 0; u < F; ++u) {
                constexpr int LAST = F - 1;
#pragma unroll
                for (int e = 0; e < V; ++e) win[(u + LAST) % F][e] = fp_pair(next[u][e], next[u][e]);
                piece.column(k + u + F + LAST, next[u]);
                const unsigned long long d[2] = {fp_pair(dyn[u].x, dyn[u].y), fp_pair(dyn[u].z, dyn[u].w)};
                dyn[u] = load(k + u + F);
                if (k + u >= piece.len) continue;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
#pragma unroll
                    for (int j = 0; j < F; ++j)
#pragma unroll
                        for (int i = 0; i < RP; ++i)
#pragma unroll
                            for (int c = 0; c < CIN; ++c) fp_fma2(acc[(i * F + j) * CIN + c][h], win[(u + j) % F][i * CIN + c], d[h]);
                    if (R0 == 0) acc[KN][h] = fp_add2(acc[KN][h], d[h]);
                }
            }
    }
    const int width = g.lanes * 4;                           // [group][k][lanes x 4 channels]
    if (!idle)
#pragma unroll
        for (int k = 0; k < NV; ++k)
            *reinterpret_cast<float4*>(red + (size_t)(grp * NV + k) * width + d0) = make_float4(fp_lo(acc[k][0]), fp_hi(acc[k][0]), fp_lo(acc[k][1]), fp_hi(acc[k][1]));
    __syncthreads();
    float* out = part + (size_t)cta * (K + 1) * g.Cout;
    for (int e = threadIdx.x; e < (R0 == 0 ? NV : KN) * g.Cout; e += FP_THREADS) {
        const int k = e / g.Cout, d = e - k * g.Cout;
        const float* r = red + k * width + d;
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
        int q = 0;
        for (; q + 4 <= g.groups; q += 4)
#pragma unroll
            for (int u = 0; u < 4; ++u) sum[u] += r[(q + u) * NV * width];
        for (; q < g.groups; ++q) sum[0] += r[q * NV * width];
        out[(size_t)(k < KN ? R0 * F * CIN + k : K) * g.Cout + d] = (sum[0] + sum[1]) + (sum[2] + sum[3]);
    }
}

template <int CIN, int F>
__global__ void __launch_bounds__(FP_THREADS, fp_ctas(CIN * F * fd_rows(CIN, F))) first_fp32_dw_kernel(const FirstWalk g, const float* __restrict__ dy, float* __restrict__ part) {
    constexpr int PARTS = F / fd_rows(CIN, F);
    extern __shared__ __align__(16) float fd_red[];
    pdl_wait();
    const int cta = blockIdx.x / PARTS, ctas = gridDim.x / PARTS, row = blockIdx.x - cta * PARTS;
    if constexpr (PARTS == 1) {
        first_dw_rows<CIN, F, 0>(g, dy, part, cta, ctas, fd_red);
    } else {
        if (row == 0) first_dw_rows<CIN, F, 0>(g, dy, part, cta, ctas, fd_red);
        if (row == 1) first_dw_rows<CIN, F, 1>(g, dy, part, cta, ctas, fd_red);
        if (row == 2) first_dw_rows<CIN, F, 2>(g, dy, part, cta, ctas, fd_red);
        if constexpr (PARTS > 3) {
            if (row == 3) first_dw_rows<CIN, F, 3>(g, dy, part, cta, ctas, fd_red);
            if (row == 4) first_dw_rows<CIN, F, 4>(g, dy, part, cta, ctas, fd_red);
        }
    }
}

// ---------------------------------------------------------------------------------- host
bool first_fp32_eligible(const AetherConvDesc& d) {
    int Ho, Wo;
    conv_out_hw(d, Ho, Wo);
    return d.Cin <= 4 && d.fH == d.fW && (d.fH == 3 || d.fH == 5) && d.sW == 1 && d.Cout <= 256 && 1LL * d.S * Ho * Wo <= 0x40000000LL;      // (pieces: 32 bits)
}
// Pieces: a row, or as many equal ones of it as make the longest walk shortest (a piece starts with a round trip to memory, some three pixels long).
// Returns the CTAs (of `most`).
static int first_walk(const AetherConvDesc& d, const float* x, int most, FirstWalk& g, unsigned* steps = nullptr) {
    g.x = x; g.S = d.S; g.H = d.H; g.W = d.W; g.sH = d.sH; g.pH = d.padH; g.pW = d.padW;
    conv_out_hw(d, g.Ho, g.Wo);
    g.Cout = d.Cout;
    g.lanes = ceil_div(d.Cout, 4);
    g.groups = FP_THREADS / g.lanes;
    const unsigned rows = (unsigned)d.S * g.Ho, room = (unsigned)most * g.groups;
    unsigned best = ~0u;
    for (int segs = 1; segs <= 8 && segs <= g.Wo; ++segs) {
        const int T = ceil_div(g.Wo, segs);
        if (segs > 1 && ceil_div(g.Wo, T) != segs) continue;
        const unsigned rounds = (rows * segs + room - 1) / room, cost = rounds * (ceil_div(T, d.fW) * d.fW + 3);        // (at most twice the pixels and a round)
        if (cost < best) { best = cost; g.segs = segs; g.T = T; }
        if (T <= d.fW) break;
    }
    if (steps) *steps = best;
    g.units = (int)(rows * g.segs);
    const int ctas = ceil_div(g.units, g.groups);
    return ctas < most ? ctas : most;
}

// (The filter in registers.  256 channels leave four pieces to a CTA: 60 x 50x50 2->256 56 us in smallc_fwd_kernel, 67 here, 40 x 64x64 3->256 82 / 85.)
bool first_fp32_fwd_eligible(const AetherConvDesc& d) {
    const int K = d.Cin * d.fH * d.fW;
    return first_fp32_eligible(d) && K <= 27 && (K <= 9 || d.Cout < 256);
}

template <int CIN, int F>
static int launch_first_fwd(const AetherConvDesc& d, const float* x, const float* w, const float* b, float* y, cudaStream_t st) {
    FirstWalk g;
    const int ctas = first_walk(d, x, num_sms() * fp_ctas(CIN * F * F), g);
    launch(first_fp32_fwd_kernel<CIN, F>, ctas, FP_THREADS, 0, st, g, w, b, y);
    count_launch();
    return check_launch("first_fp32_fwd_kernel");
}

static int first_dw_most(const AetherConvDesc& d) {
    const int rows = fd_rows(d.Cin, d.fH);
    return num_sms() * fp_ctas(d.Cin * d.fW * rows) / (d.fH / rows);
}
// Against the kernels that took these layers before (us): smallc_dw_kernel 10 and a product in 1/15 or, of up to 64 values, 1/6.8 ps, the GEMM of simt_dw_kernel 10 and
// a product of its tiles in 1/14 ps, 1/23 of four input channels.  Here a step of all pieces takes 10.7 ns per value, half of that where two CTAs share an SM, unless
// dy, read again by every row of a filter of more than 27 values, takes longer (3.1 TB/s), and the sums of a CTA meet in 1.65 ns per value and thread.  (us, there /
// here: 300 x 16x18 4->256 5x5 123 / 213, 100 x 28x28 4->128 5x5 62 / 104, 84 x 116x88 2->54 5x5 227 / 422, 60 x 64x64 3->208 167 / 155, 128 x 56x56 1->224
// 5x5 226 / 193.  Over 972 layers at most 38 % behind the faster one, 1.0 % in the mean, here everywhere 86 and 2.7 %.  Few values or channels: always here.)
bool first_fp32_dw_eligible(const AetherConvDesc& d) {
    if (!first_fp32_eligible(d)) return false;
    const int K = d.Cin * d.fH * d.fW, rows = fd_rows(d.Cin, d.fH), values = d.Cin * d.fW * rows;
    if (K < 25 || d.Cout <= 32) return true;
    FirstWalk g;
    unsigned steps;
    first_walk(d, nullptr, first_dw_most(d), g, &steps);
    const double pixels = 1.0 * d.S * g.Ho * g.Wo, ragged = d.Cout % 4 ? 1.0 : 0.0;
    const double walk = steps * values * (fp_ctas(values) == 2 ? 5.6e-3 : 10.7e-3) * (1.0 + 0.14 * ragged);
    const double reads = d.fH / rows * pixels * d.Cout * 4.0 * 0.32e-6 * (1.0 + 0.26 * ragged);
    const double here = 5.4 + (walk > reads ? walk : reads) + g.lanes * K * 1.65e-3;
    const double there = smallc_conv_eligible(d) ? 10.0 + pixels * K * d.Cout * (K > 64 ? 1e-6 / 15.0 : 1e-6 / 6.8)
                                                 : 10.0 + pixels * (ceil_div(K, 32) * 32) * (ceil_div(d.Cout, 64) * 64) * (d.Cin == 4 && !ragged ? 1e-6 / 23.0 : 1e-6 / 14.0);
    return here < there;
}
// Against first_tc_bwd_filter without a copy of dy: 10.5 products a nanosecond here, 36 ns per 1000 pixels and a fixed part that is 3.5 us longer there.
// (us: 14 x 8x9 3->16 10.8 there, 6.5 here; 211 x 28x28 3->16 16.9 / 13.2, 300 x 40x40 1->16 26.0 / 14.5, 512 x 28x28 1->32 23.4 / 21; 128 x 32x32 3->32 14.3 / 14.8,
// 17 x 7x7 3->128 8.0 / 9.5.)
bool first_fp32_dw_faster(const AetherConvDesc& d) {
    int Ho, Wo;
    conv_out_hw(d, Ho, Wo);
    const int products = d.fH * d.fW * d.Cin * d.Cout;
    return products <= 512 && 1.0 * d.S * Ho * Wo * (products / 10.5 - 36.0) < 3.5e6;
}
size_t first_fp32_dw_workspace_bytes(const AetherConvDesc& d) {
    FirstWalk g;
    return align_up((size_t)first_walk(d, nullptr, first_dw_most(d), g) * (d.fH * d.fW * d.Cin + 1) * d.Cout * sizeof(float), 1024);
}

template <int CIN, int F>
static int launch_first_dw(const AetherConvDesc& d, const float* x, const float* dy, float* dw, float* db, void* ws, size_t ws_bytes, cudaStream_t st) {
    constexpr int NV = fd_rows(CIN, F) * F * CIN + 1;
    FirstWalk g;
    const int ctas = first_walk(d, x, first_dw_most(d), g);
    const size_t need = (size_t)ctas * (CIN * F * F + 1) * d.Cout * sizeof(float);
    if (!ws || ws_bytes < need) return set_error(AE_BAD_ARG, "conv workspace too small: %zu < %zu", ws_bytes, need);
    static PerDeviceSmem once;
    if (int rc = ensure_dynamic_smem(first_fp32_dw_kernel<CIN, F>, FP_THREADS * 16 * NV, once, "first_fp32_dw_kernel")) return rc;
    launch(first_fp32_dw_kernel<CIN, F>, ctas * (F / fd_rows(CIN, F)), FP_THREADS, g.groups * g.lanes * 16 * NV, st, g, dy, static_cast<float*>(ws));
    count_launch();
    if (int rc = check_launch("first_fp32_dw_kernel")) return rc;
    return smallc_reduce_partials(static_cast<float*>(ws), ctas, CIN * F * F, d.Cout, dw, db, st);
}

int first_fp32_fwd(const AetherConvDesc& d, const float* x, const float* w, const float* b, float* y, cudaStream_t st) {
    if (d.fH == 5) return launch_first_fwd<1, 5>(d, x, w, b, y, st);
    return d.Cin == 1 ? launch_first_fwd<1, 3>(d, x, w, b, y, st) : d.Cin == 2 ? launch_first_fwd<2, 3>(d, x, w, b, y, st) : launch_first_fwd<3, 3>(d, x, w, b, y, st);
}

int first_fp32_bwd_filter(const AetherConvDesc& d, const float* x, const float* dy, float* dw, float* db, void* ws, size_t ws_bytes, cudaStream_t st) {
    const bool five = d.fH == 5;
    switch (d.Cin) {
        case 1: return five ? launch_first_dw<1, 5>(d, x, dy, dw, db, ws, ws_bytes, st) : launch_first_dw<1, 3>(d, x, dy, dw, db, ws, ws_bytes, st);
        case 2: return five ? launch_first_dw<2, 5>(d, x, dy, dw, db, ws, ws_bytes, st) : launch_first_dw<2, 3>(d, x, dy, dw, db, ws, ws_bytes, st);
        case 3: return five ? launch_first_dw<3, 5>(d, x, dy, dw, db, ws, ws_bytes, st) : launch_first_dw<3, 3>(d, x, dy, dw, db, ws, ws_bytes, st);
        default: return five ? launch_first_dw<4, 5>(d, x, dy, dw, db, ws, ws_bytes, st) : launch_first_dw<4, 3>(d, x, dy, dw, db, ws, ws_bytes, st);
    }
}

}  // namespace aether
