// fp32 CUDA-core convolution for every filter size / stride / padding Conv_Layer accepts
// (CNN/models/CNN_classes_cupy.py:70-154).  It serves the shapes the tensor-core kernels do not
// take: the first layers with 1 or 3 input channels (HBM-bound, a few FLOP per byte), strided
// convolutions, channel counts that are not a multiple of 4, and AETHER_MATH_FP32.
#include "common.cuh"
#include "tc_host.cuh"

namespace aether {

// Pointwise layers with very few outputs per pixel (a classifier head: Dense 1024 -> 10 is a 1x1 convolution with
// Cout = 10): with one thread per output element a batch of 512 rows is 5120 threads walking 1024 channels each.
// Here a warp takes a row: the lanes split the channels (float4 loads of x, the row is read once), keep Cout partial
// sums each and combine them with shuffles in a fixed order.
// The filter is kept transposed in shared memory, wT[d][Cin], so a lane's four channels of output d are one 16-byte
// shared-memory read (4 * Cout scalar global loads per four channels before).
// (rows of Cin + 4 floats: with Cin a multiple of 32 the outputs of one channel would all fall on one bank)
__device__ __forceinline__ void head_load_filter_T(const float* __restrict__ w, float* wT, int Cin, int Cout) {
    for (int i = threadIdx.x; i < Cin * Cout; i += blockDim.x) {
        const int c = i / Cout, d = i - c * Cout;
        wT[d * (Cin + 4) + c] = w[i];
    }
    __syncthreads();
}

template <int MAXD>
__global__ void __launch_bounds__(256) gen_fwd_pointwise_few_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                                    const float* __restrict__ b, float* __restrict__ y,
                                                                    long long rows, int Cin, int Cout) {
    pdl_wait();
    extern __shared__ __align__(16) float head_wT[];
    head_load_filter_T(w, head_wT, Cin, Cout);
    const int lane = threadIdx.x & 31;
    const long long warp0 = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    const int C4 = Cin >> 2;
    for (long long row = warp0; row < rows; row += nwarps) {
        float acc[MAXD];
#pragma unroll
        for (int d = 0; d < MAXD; ++d) acc[d] = 0.f;
        const float4* xr = reinterpret_cast<const float4*>(x + (size_t)row * Cin);
        for (int c4 = lane; c4 < C4; c4 += 32) {
            const float4 v = xr[c4];
#pragma unroll
            for (int d = 0; d < MAXD; ++d) {
                if (d < Cout) {
                    const float4 k = *reinterpret_cast<const float4*>(head_wT + d * (Cin + 4) + 4 * c4);
                    acc[d] = fmaf(v.x, k.x, fmaf(v.y, k.y, fmaf(v.z, k.z, fmaf(v.w, k.w, acc[d]))));
                }
            }
        }
#pragma unroll
        for (int d = 0; d < MAXD; ++d) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc[d] += __shfl_xor_sync(0xffffffffu, acc[d], o);
        }
        if (lane < Cout) {
            float r = 0.f;
#pragma unroll
            for (int d = 0; d < MAXD; ++d) r = (d == lane) ? acc[d] : r;
            y[(size_t)row * Cout + lane] = r + (b ? b[lane] : 0.f);
        }
    }
}

// ---------------------------------------------------------------------------------- dX of first layers
// dx[s,h,w,c] = sum over taps (i,j) and d of dy[s,ho,wo,d] * w[i,j,c,d] with ho*sH + i - pH == h.
//
// Layers with 1..4 input channels and a filter count that is a multiple of 4 (the first layer of a
// network): one thread per input pixel keeps all CIN sums, so every dy vector is loaded once as float4 and the
// filter reads are the same address for the whole warp.
template <int CIN>
__global__ void __launch_bounds__(256) gen_dx_fewc_kernel(const float* __restrict__ dy, const float* __restrict__ w,
                                                          float* __restrict__ dx, int S, int H, int W, int Cout, int fH,
                                                          int fW, int sH, int sW, int pH, int pW, int Ho, int Wo) {
    pdl_wait();
    const long long total = 1LL * S * H * W;
    const int C4 = Cout >> 2;
    for (long long pix = blockIdx.x * (long long)blockDim.x + threadIdx.x; pix < total;
         pix += (long long)gridDim.x * blockDim.x) {
        const int wi = (int)(pix % W);
        const long long q = pix / W;
        const int hi = (int)(q % H);
        const int s = (int)(q / H);
        float acc[CIN];
#pragma unroll
        for (int c = 0; c < CIN; ++c) acc[c] = 0.f;
        for (int i = 0; i < fH; ++i) {
            const int hn = hi + pH - i;
            if (hn < 0 || hn % sH) continue;
            const int ho = hn / sH;
            if (ho >= Ho) continue;
            for (int j = 0; j < fW; ++j) {
                const int wn = wi + pW - j;
                if (wn < 0 || wn % sW) continue;
                const int wo = wn / sW;
                if (wo >= Wo) continue;
                const float4* dyp = reinterpret_cast<const float4*>(dy + (((size_t)s * Ho + ho) * Wo + wo) * Cout);
                const float4* wq = reinterpret_cast<const float4*>(w + (size_t)(i * fW + j) * CIN * Cout);
#pragma unroll 4
                for (int d = 0; d < C4; ++d) {
                    const float4 g = dyp[d];
#pragma unroll
                    for (int c = 0; c < CIN; ++c) {
                        const float4 k = __ldg(wq + c * C4 + d);
                        acc[c] = fmaf(g.x, k.x, fmaf(g.y, k.y, fmaf(g.z, k.z, fmaf(g.w, k.w, acc[c]))));
                    }
                }
            }
        }
#pragma unroll
        for (int c = 0; c < CIN; ++c) dx[pix * CIN + c] = acc[c];
    }
}

// ---------------------------------------------------------------------------------- classifier heads, backward
// dx[p][c] = sum_d dy[p][d] * w[c][d] for a pointwise layer with few outputs: a block takes a row at a time, a thread
// four channels; the filter is read transposed from shared memory, the row of dy is the same address for every thread.
template <int MAXD>
__global__ void __launch_bounds__(256) head_dx_kernel(const float* __restrict__ dy, const float* __restrict__ w,
                                                      float* __restrict__ dx, long long rows, int Cin, int Cout) {
    pdl_wait();
    extern __shared__ __align__(16) float head_wT[];
    head_load_filter_T(w, head_wT, Cin, Cout);
    const int C4 = Cin >> 2;
    float gn[MAXD];                                     // the next row's dy values, requested one row ahead
#pragma unroll
    for (int d = 0; d < MAXD; ++d) gn[d] = (d < Cout && blockIdx.x < rows) ? __ldg(dy + (size_t)blockIdx.x * Cout + d) : 0.f;
    for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
        float g[MAXD];
        const long long nrow = row + gridDim.x;
#pragma unroll
        for (int d = 0; d < MAXD; ++d) {
            g[d] = gn[d];
            gn[d] = (d < Cout && nrow < rows) ? __ldg(dy + (size_t)nrow * Cout + d) : 0.f;
        }
        float4* out = reinterpret_cast<float4*>(dx + (size_t)row * Cin);
        for (int c4 = threadIdx.x; c4 < C4; c4 += blockDim.x) {
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int d = 0; d < MAXD; ++d) {
                if (d < Cout) {
                    const float4 k = *reinterpret_cast<const float4*>(head_wT + d * (Cin + 4) + 4 * c4);
                    a.x = fmaf(g[d], k.x, a.x); a.y = fmaf(g[d], k.y, a.y); a.z = fmaf(g[d], k.z, a.z); a.w = fmaf(g[d], k.w, a.w);
                }
            }
            out[c4] = a;
        }
    }
}

// dw[c][d] = sum_p x[p][c] * dy[p][d], db[d] = sum_p dy[p][d] over a part of the rows: partials [part][Cout + 1][Cin]
// (row Cout: the column sums of dy), d-major so that the threads' stores are whole lines, that head_dw_reduce_kernel adds up.  A thread keeps four channels x Cout sums; x is read once, coalesced; the row of dy
// is the same address for every thread of a row.  A block is row lanes x four-channel groups (blockIdx.y walks the
// groups beyond 256) and every row lane writes a part of its own.  Few rows per thread: the loop is a chain of load
// latencies (4 blocks of 32 rows at batch 128 took 17 us, of which the sums themselves are a small part).
template <int MAXD>
__global__ void __launch_bounds__(256) head_dw_partial_kernel(const float* __restrict__ x, const float* __restrict__ dy,
                                                              float* __restrict__ part, long long rows, int Cin, int Cout,
                                                              int lanes, int parts) {
    pdl_wait();
    const int C4 = Cin >> 2;
    const int groups = 256 / lanes;
    const int rl = threadIdx.x / groups, gi = threadIdx.x - rl * groups;
    const int c4 = blockIdx.y * groups + gi;
    const int mine = blockIdx.x * lanes + rl;             // this row lane's part: rows mine, mine + parts, ...
    if (rl >= lanes || mine >= parts) return;
    float* out = part + (size_t)mine * (Cout + 1) * Cin;
    if (c4 < C4) {
        float4 acc[MAXD];
#pragma unroll
        for (int d = 0; d < MAXD; ++d) acc[d] = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4* xp = reinterpret_cast<const float4*>(x) + c4;
#pragma unroll 4
        for (long long r = mine; r < rows; r += parts) {
            const float4 v = xp[(size_t)r * C4];
            const float* gr = dy + (size_t)r * Cout;
#pragma unroll
            for (int d = 0; d < MAXD; ++d) {
                if (d < Cout) {
                    const float g = __ldg(gr + d);
                    acc[d].x = fmaf(v.x, g, acc[d].x); acc[d].y = fmaf(v.y, g, acc[d].y);
                    acc[d].z = fmaf(v.z, g, acc[d].z); acc[d].w = fmaf(v.w, g, acc[d].w);
                }
            }
        }
#pragma unroll
        for (int d = 0; d < MAXD; ++d)
            if (d < Cout) *reinterpret_cast<float4*>(out + (size_t)d * Cin + 4 * c4) = acc[d];
    }
    if (blockIdx.y == 0 && gi < Cout) {
        float sdy = 0.f;
#pragma unroll 4
        for (long long r = mine; r < rows; r += parts) sdy += dy[(size_t)r * Cout + gi];
        out[(size_t)Cout * Cin + gi] = sdy;
    }
}

// dw[c][d] = sum over parts of part[p][d][c], db[d] of part[p][Cout][d]: 32 outputs x 8 lanes per block, fixed order.
__global__ void __launch_bounds__(256) head_dw_reduce_kernel(const float* __restrict__ part, int parts, int Cin, int Cout,
                                                             float* __restrict__ dw, float* __restrict__ db) {
    pdl_wait();
    __shared__ float red[8][32];
    const int el = threadIdx.x & 31, ln = threadIdx.x >> 5;
    const int e = blockIdx.x * 32 + el, total = Cin * Cout + Cout;        // d-major, then the Cout column sums
    float s = 0.f;
    if (e < total)
#pragma unroll 4
        for (int p = ln; p < parts; p += 8) s += part[(size_t)p * (Cout + 1) * Cin + e];
    red[ln][el] = s;
    __syncthreads();
    if (ln == 0 && e < total) {
        float t = 0.f;
#pragma unroll
        for (int l = 0; l < 8; ++l) t += red[l][el];
        if (e < Cin * Cout) {
            const int d = e / Cin, c = e - d * Cin;
            if (dw) dw[c * Cout + d] = t;
        } else if (db) {
            db[e - Cin * Cout] = t;
        }
    }
}

// Pointwise layer with at most 16 outputs whose transposed filter fits in shared memory (a classifier head).
static bool head_shape(const AetherConvDesc& d) {
    return d.fH == 1 && d.fW == 1 && d.sH == 1 && d.sW == 1 && d.padH == 0 && d.padW == 0 && d.Cout <= 16 && d.Cin >= 128 &&
           (d.Cin & 3) == 0 && (size_t)(d.Cin + 4) * d.Cout * sizeof(float) <= 96 * 1024;
}

// ---------------------------------------------------------------------------------- host
static int gen_blocks(long long total, int threads) {
    long long b = (total + threads - 1) / threads;
    const long long cap = 148LL * 16;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (int)b;
}

int generic_conv_fwd(const AetherConvDesc& d, const float* x, const float* w, const float* b, float* y, cudaStream_t st) {
    if (head_shape(d) && (reinterpret_cast<uintptr_t>(x) & 15u) == 0) {
        const long long rows = 1LL * d.S * d.H * d.W;
        const int smem = (d.Cin + 4) * d.Cout * (int)sizeof(float);
        static PerDeviceSmem configured;
        if (int rc = ensure_dynamic_smem(gen_fwd_pointwise_few_kernel<16>, 96 * 1024, configured, "head forward")) return rc;
        long long nb = (rows + 7) / 8;                        // a warp per row, 8 rows per block and pass
        if (nb > 2LL * num_sms()) nb = 2LL * num_sms();       // every block loads the filter once
        launch(gen_fwd_pointwise_few_kernel<16>, (int)nb, 256, smem, st, x, w, b, y, rows, d.Cin, d.Cout);
        count_launch();
        return check_launch("gen_fwd_pointwise_few_kernel");
    }
    return simt_conv_fwd(d, x, w, b, y, st);
}

int generic_conv_bwd_data(const AetherConvDesc& d, const float* dy, const float* w, float* dx, cudaStream_t st) {
    int Ho, Wo;
    conv_out_hw(d, Ho, Wo);
    if (d.Cin <= 4 && d.Cout % 4 == 0 && (reinterpret_cast<uintptr_t>(dy) & 15u) == 0 && (reinterpret_cast<uintptr_t>(w) & 15u) == 0) {
        const int nb = gen_blocks(1LL * d.S * d.H * d.W, 256);
#define AETHER_DX_FEWC(CIN)                                                                                          \
    launch(gen_dx_fewc_kernel<CIN>, nb, 256, 0, st, dy, w, dx, d.S, d.H, d.W, d.Cout, d.fH, d.fW, d.sH, d.sW, d.padH, d.padW, Ho, Wo)
        switch (d.Cin) {
            case 1: AETHER_DX_FEWC(1); break;
            case 2: AETHER_DX_FEWC(2); break;
            case 3: AETHER_DX_FEWC(3); break;
            default: AETHER_DX_FEWC(4); break;
        }
#undef AETHER_DX_FEWC
        count_launch();
        return check_launch("gen_dx_fewc_kernel");
    }
    if (head_shape(d) && (reinterpret_cast<uintptr_t>(dx) & 15u) == 0) {
        const long long rows = 1LL * d.S * d.H * d.W;
        const int smem = (d.Cin + 4) * d.Cout * (int)sizeof(float);
        static PerDeviceSmem configured;
        if (int rc = ensure_dynamic_smem(head_dx_kernel<16>, 96 * 1024, configured, "head dX")) return rc;
        long long nb = rows < 2LL * num_sms() ? rows : 2LL * num_sms();
        launch(head_dx_kernel<16>, (int)nb, 256, smem, st, dy, w, dx, rows, d.Cin, d.Cout);
        count_launch();
        return check_launch("head_dx_kernel");
    }
    return simt_conv_bwd_data(d, dy, w, dx, st);
}

// Parts of the rows of a classifier head's dW: four rows each until there are 128 of them (their sum is a pass of its own).
static int head_dw_parts(const AetherConvDesc& d) {
    const long long rows = 1LL * d.S * d.H * d.W, n = (rows + 3) / 4;
    return (int)(n < 128 ? n : 128);
}

size_t generic_conv_workspace_bytes(const AetherConvDesc& d) {
    const size_t simt = simt_conv_workspace_bytes(d);
    if (!head_shape(d)) return simt;
    const size_t head = align_up((size_t)head_dw_parts(d) * (d.Cout + 1) * d.Cin * sizeof(float), 1024);
    return head > simt ? head : simt;
}

int generic_conv_bwd_filter(const AetherConvDesc& d, const float* x, const float* dy, float* dw, float* db, void* ws,
                            size_t ws_bytes, cudaStream_t st) {
    if (!head_shape(d) || x == nullptr || (reinterpret_cast<uintptr_t>(x) & 15u)) return simt_conv_bwd_filter(d, x, dy, dw, db, ws, ws_bytes, st);
    if (!ws || ws_bytes < generic_conv_workspace_bytes(d))
        return set_error(AE_BAD_ARG, "conv workspace too small: %zu < %zu", ws_bytes, generic_conv_workspace_bytes(d));
    const int parts = head_dw_parts(d), C4 = d.Cin / 4;
    int lanes = 1;                                       // row lanes per block: as many as whole channel rows fit 256 threads
    while (lanes * 2 <= parts && C4 * lanes * 2 <= 256) lanes *= 2;
    const int groups = 256 / lanes;
    float* part = static_cast<float*>(ws);
    launch(head_dw_partial_kernel<16>, dim3(ceil_div(parts, lanes), ceil_div(C4, groups)), 256, 0, st, x, dy, part, 1LL * d.S * d.H * d.W, d.Cin,
           d.Cout, lanes, parts);
    count_launch();
    if (int rc = check_launch("head_dw_partial_kernel")) return rc;
    launch(head_dw_reduce_kernel, ceil_div((d.Cin + 1) * d.Cout, 32), 256, 0, st, part, parts, d.Cin, d.Cout, dw, db);
    count_launch();
    return check_launch("head_dw_reduce_kernel");
}

}  // namespace aether
