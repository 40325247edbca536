// Single-precision convolution (CNN/models/CNN_classes_cupy.py:70-154) for the shapes the tensor-core kernels do not take:
// classifier heads (pointwise layers with few outputs per pixel) and the dX of first layers (1 to 4 input channels) have
// kernels of their own here, everything else goes to the tiled implicit GEMMs of conv_simt.cu.
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
                                                                    long long rows, int Cin, int Cout, float* __restrict__ prob) {
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
        float z = -INFINITY;
        if (lane < Cout) {
            float r = 0.f;
#pragma unroll
            for (int d = 0; d < MAXD; ++d) r = (d == lane) ? acc[d] : r;
            z = r + (b ? b[lane] : 0.f);
            y[(size_t)row * Cout + lane] = z;
        }
        if (prob != nullptr) {                               // the softmax behind the head, as softmax_cce_kernel computes it
            float mx = z;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const float e = lane < Cout ? expf(z - mx) : 0.f;
            float sum = e;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            if (lane < Cout) prob[(size_t)row * Cout + lane] = e / sum;
        }
    }
}

// ---------------------------------------------------------------------------------- dX of first layers
// dx[s,h,w,c] = sum over taps (i,j) and d of dy[s,ho,wo,d] * w[i,j,c,d] with ho*sH + i - pH == h, for layers with 1..4
// input channels (the first layer of a network), always in single precision.
//
// Bound by the FMA pipes and the L1: dy is small and every value of it meets CIN * taps filter values.  Eight lanes
// share a column of four input pixels and take four output channels each, so a warp's load of dy is four whole
// 128-byte lines, and a load of dy serves up to FB taps of the filter column (FB rows of the filter sit in registers at a
// time: 3x3 filters read each dy value 1.5 times per column instead of three times).  Sums are pairs over even and odd
// channels (fma.rn.f32x2), the lanes' sums meet in a fixed halving exchange.  A stride splits the input pixels into
// sH*sW classes (blockIdx.z) that each see only the taps that reach them.
// Measured: 128 x 32x32 3->32 3x3, 56 us with one thread per pixel (a warp's load touched 32 lines), 20 us now.
static constexpr int DXF_PV = 4;                        // pixels (rows) per thread
static constexpr int DXF_LANES = 8;                     // lanes that share them

__device__ __forceinline__ void dxf_fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

// Four consecutive floats of an array as two pairs; of an unaligned row the n that are in it.
template <bool VEC>
__device__ __forceinline__ ulonglong2 dxf_load4(const float* p, int n) {
    if (VEC) return __ldg(reinterpret_cast<const ulonglong2*>(p));
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (n > 0) v.x = __ldg(p);
    if (n > 1) v.y = __ldg(p + 1);
    if (n > 2) v.z = __ldg(p + 2);
    if (n > 3) v.w = __ldg(p + 3);
    ulonglong2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.x) : "f"(v.x), "f"(v.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.y) : "f"(v.z), "f"(v.w));
    return r;
}

template <int CIN, int FB, bool VEC>
__global__ void __launch_bounds__(256, 2) dx_fewc_kernel(const float* __restrict__ dy, const float* __restrict__ w, float* __restrict__ dx,
                                                         int S, int H, int W, int Cout, int fH, int fW, int sH, int sW, int pH, int pW,
                                                         int Ho, int Wo) {
    pdl_wait();
    constexpr int PV = DXF_PV;
    // this class: rows h = hs + a * sH, taps i = ph + sH * ti, dy row a + hq - ti (columns alike)
    const int ph = blockIdx.z / sW, pw = blockIdx.z - ph * sW;
    const int nH = ph < fH ? (fH - ph - 1) / sH + 1 : 0, nW = pw < fW ? (fW - pw - 1) / sW + 1 : 0;
    const int hs = ((ph - pH) % sH + sH) % sH, ws = ((pw - pW) % sW + sW) % sW;
    const int hq = (hs + pH - ph) / sH, wq = (ws + pW - pw) / sW;
    const int MH = hs < H ? (H - hs - 1) / sH + 1 : 0, MW = ws < W ? (W - ws - 1) / sW + 1 : 0;
    if (MH == 0 || MW == 0) return;
    const int strips = (MH + PV - 1) / PV;
    const long long items = 1LL * S * strips * MW;
    const long long item = blockIdx.x * (256LL / DXF_LANES) + threadIdx.x / DXF_LANES;
    const bool live = item < items;                     // (every lane takes part in the exchange below)
    const int sub = threadIdx.x % DXF_LANES;
    int b, a0;
    long long s;
    if (items < 1LL << 31) {
        const unsigned it = live ? (unsigned)item : 0u, q = it / (unsigned)MW;
        b = (int)(it - q * MW);
        const unsigned s32 = q / (unsigned)strips;
        a0 = (int)(q - s32 * strips) * PV;
        s = s32;
    } else {
        const long long it = live ? item : 0, q = it / MW;
        b = (int)(it - q * MW);
        s = q / strips;
        a0 = (int)(q - s * strips) * PV;
    }

    unsigned long long acc[PV][CIN];
#pragma unroll
    for (int p = 0; p < PV; ++p)
#pragma unroll
        for (int c = 0; c < CIN; ++c) acc[p][c] = 0ull;
    const float* dys = dy + s * Ho * Wo * Cout;
#pragma unroll 1
    for (int ti0 = 0; ti0 < nH; ti0 += FB) {            // (FB divides nH)
        const int r0 = a0 + hq - ti0 - (FB - 1);        // dy row of the first load
#pragma unroll 1
        for (int tj = 0; tj < nW; ++tj) {
            const int wo = b + wq - tj;
            if (!live || (unsigned)wo >= (unsigned)Wo) continue;
#pragma unroll 1
            for (int d = sub * 4; d < Cout; d += DXF_LANES * 4) {
                ulonglong2 k[FB][CIN], v[PV + FB - 1];
#pragma unroll
                for (int r = 0; r < PV + FB - 1; ++r) {
                    const int ho = r0 + r;
                    v[r] = (unsigned)ho < (unsigned)Ho ? dxf_load4<VEC>(dys + ((long long)ho * Wo + wo) * Cout + d, Cout - d) : make_ulonglong2(0ull, 0ull);
                }
                const float* wt = w + ((long long)(ph + ti0 * sH) * fW + pw + tj * sW) * CIN * Cout + d;
#pragma unroll
                for (int t = 0; t < FB; ++t)
#pragma unroll
                    for (int c = 0; c < CIN; ++c) k[t][c] = dxf_load4<VEC>(wt + ((long long)t * sH * fW * CIN + c) * Cout, Cout - d);
#pragma unroll
                for (int p = 0; p < PV; ++p)
#pragma unroll
                    for (int t = 0; t < FB; ++t)
#pragma unroll
                        for (int c = 0; c < CIN; ++c) {
                            dxf_fma2(acc[p][c], v[p + FB - 1 - t].x, k[t][c].x);
                            dxf_fma2(acc[p][c], v[p + FB - 1 - t].y, k[t][c].y);
                        }
            }
        }
    }

    // Eight lanes' sums of four pixels: two exchanges that halve the pixels a lane keeps, one that adds.
    float f[PV][CIN];
#pragma unroll
    for (int p = 0; p < PV; ++p)
#pragma unroll
        for (int c = 0; c < CIN; ++c) f[p][c] = __uint_as_float((unsigned)acc[p][c]) + __uint_as_float((unsigned)(acc[p][c] >> 32));
    const bool hi4 = sub & 4, hi2 = sub & 2;
#pragma unroll
    for (int c = 0; c < CIN; ++c) {
        const float s0 = __shfl_xor_sync(0xffffffffu, hi4 ? f[0][c] : f[2][c], 4), s1 = __shfl_xor_sync(0xffffffffu, hi4 ? f[1][c] : f[3][c], 4);
        const float u0 = (hi4 ? f[2][c] : f[0][c]) + s0, u1 = (hi4 ? f[3][c] : f[1][c]) + s1;
        const float s2 = __shfl_xor_sync(0xffffffffu, hi2 ? u0 : u1, 2);
        const float u = (hi2 ? u1 : u0) + s2;
        f[0][c] = u + __shfl_xor_sync(0xffffffffu, u, 1);
    }
    const int a = a0 + (sub >> 1);
    if (live && !(sub & 1) && a < MH) {
        float* o = dx + ((s * H + hs + (long long)a * sH) * W + ws + (long long)b * sW) * CIN;
#pragma unroll
        for (int c = 0; c < CIN; ++c) o[c] = f[0][c];
    }
}

// ---------------------------------------------------------------------------------- classifier heads, backward
// dx[p][c] = sum_d dy[p][d] * w[c][d] for a pointwise layer with few outputs: a block takes a row at a time, a thread
// four channels; the filter is read transposed from shared memory, the row of dy is the same address for every thread.
// CCE: dy is not there yet -- it is the combined softmax / cross-entropy gradient (prob - y_smooth) / rows, which is computed
// from the probabilities and the labels of the row (as softmax_cce_kernel does) and written to dz on the way.
struct HeadCce {
    const float* prob;
    const int* labels;             // one of the three
    const long long* labels64;
    const float* targets;
    float* dz;
    float smooth, inv_rows;
};
template <int MAXD, bool CCE>
__global__ void __launch_bounds__(256) head_dx_kernel(const float* __restrict__ dy, const float* __restrict__ w,
                                                      float* __restrict__ dx, long long rows, int Cin, int Cout, const HeadCce cce) {
    pdl_wait();
    extern __shared__ __align__(16) float head_wT[];
    head_load_filter_T(w, head_wT, Cin, Cout);
    const int C4 = Cin >> 2;
    const float* src = CCE ? cce.prob : dy;
    float gn[MAXD];                                     // the next row's dy values, requested one row ahead
#pragma unroll
    for (int d = 0; d < MAXD; ++d) gn[d] = (d < Cout && blockIdx.x < rows) ? __ldg(src + (size_t)blockIdx.x * Cout + d) : 0.f;
    for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
        float g[MAXD];
        const long long nrow = row + gridDim.x;
#pragma unroll
        for (int d = 0; d < MAXD; ++d) {
            g[d] = gn[d];
            gn[d] = (d < Cout && nrow < rows) ? __ldg(src + (size_t)nrow * Cout + d) : 0.f;
        }
        if (CCE) {
            const int label = cce.labels ? cce.labels[row] : cce.labels64 ? (int)cce.labels64[row] : -1;
#pragma unroll
            for (int d = 0; d < MAXD; ++d) {
                if (d < Cout) {
                    const float onehot = cce.targets ? cce.targets[(size_t)row * Cout + d] : (d == label ? 1.f : 0.f);
                    const float tb = onehot * (1.f - cce.smooth) + cce.smooth / Cout;
                    g[d] = (g[d] - tb) * cce.inv_rows;
                    if ((int)threadIdx.x == d) cce.dz[(size_t)row * Cout + d] = g[d];
                }
            }
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
static int head_fwd(const AetherConvDesc& d, const float* x, const float* w, const float* b, float* y, float* prob, cudaStream_t st) {
    const long long rows = 1LL * d.S * d.H * d.W;
    const int smem = (d.Cin + 4) * d.Cout * (int)sizeof(float);
    static PerDeviceSmem configured;
    if (int rc = ensure_dynamic_smem(gen_fwd_pointwise_few_kernel<16>, 96 * 1024, configured, "head forward")) return rc;
    long long nb = (rows + 7) / 8;                        // a warp per row, 8 rows per block and pass
    if (nb > 2LL * num_sms()) nb = 2LL * num_sms();       // every block loads the filter once
    launch(gen_fwd_pointwise_few_kernel<16>, (int)nb, 256, smem, st, x, w, b, y, rows, d.Cin, d.Cout, prob);
    count_launch();
    return check_launch("gen_fwd_pointwise_few_kernel");
}

int generic_conv_fwd(const AetherConvDesc& d, const float* x, const float* w, const float* b, float* y, void* ws, size_t ws_bytes,
                     cudaStream_t st) {
    if (head_shape(d) && (reinterpret_cast<uintptr_t>(x) & 15u) == 0) return head_fwd(d, x, w, b, y, nullptr, st);
    return simt_conv_fwd(d, x, w, b, y, ws, ws_bytes, st);
}

bool generic_head_shape(const AetherConvDesc& d) { return head_shape(d); }
int generic_head_softmax_fwd(const AetherConvDesc& d, const float* x, const float* w, const float* b, float* y, float* prob, cudaStream_t st) {
    return head_fwd(d, x, w, b, y, prob, st);
}

static int head_dx(const AetherConvDesc& d, const float* dy, const float* w, float* dx, const HeadCce* cce, cudaStream_t st) {
    const long long rows = 1LL * d.S * d.H * d.W;
    const int smem = (d.Cin + 4) * d.Cout * (int)sizeof(float);
    static PerDeviceSmem configured[2];
    const auto kernel = cce ? head_dx_kernel<16, true> : head_dx_kernel<16, false>;
    if (int rc = ensure_dynamic_smem(kernel, 96 * 1024, configured[cce ? 1 : 0], "head dX")) return rc;
    const long long nb = rows < 2LL * num_sms() ? rows : 2LL * num_sms();
    launch(kernel, (int)nb, 256, smem, st, dy, w, dx, rows, d.Cin, d.Cout, cce ? *cce : HeadCce{});
    count_launch();
    return check_launch("head_dx_kernel");
}
int generic_head_cce_bwd(const AetherConvDesc& d, const float* prob, const int* labels, const long long* labels64, const float* targets,
                         float smooth, const float* w, float* dz, float* dx, cudaStream_t st) {
    const HeadCce cce = {prob, labels, labels64, targets, dz, smooth, 1.f / (float)(1LL * d.S * d.H * d.W)};
    return head_dx(d, nullptr, w, dx, &cce, st);
}

template <int CIN, int FB>
static void dx_fewc_launch(const AetherConvDesc& d, const float* dy, const float* w, float* dx, int Ho, int Wo, cudaStream_t st) {
    const bool vec = d.Cout % 4 == 0 && ((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(w)) & 15u) == 0;
    const int MH = ceil_div(d.H, d.sH), MW = ceil_div(d.W, d.sW);            // extent of the largest class
    const long long items = 1LL * d.S * ceil_div(MH, DXF_PV) * MW;
    const dim3 grid((unsigned)((items + 256 / DXF_LANES - 1) / (256 / DXF_LANES)), 1, d.sH * d.sW);
    launch(vec ? dx_fewc_kernel<CIN, FB, true> : dx_fewc_kernel<CIN, FB, false>, grid, 256, 0, st, dy, w, dx, d.S, d.H, d.W, d.Cout, d.fH, d.fW,
           d.sH, d.sW, d.padH, d.padW, Ho, Wo);
}

template <int CIN>
static int dx_fewc(const AetherConvDesc& d, const float* dy, const float* w, float* dx, int Ho, int Wo, cudaStream_t st) {
    // filter rows per pass: all of the usual filters' (their CIN * rows vectors fit the registers), else one
    if (d.sH == 1 && d.fH == 3) dx_fewc_launch<CIN, 3>(d, dy, w, dx, Ho, Wo, st);
    else if (d.sH == 1 && d.fH == 5) dx_fewc_launch<CIN, 5>(d, dy, w, dx, Ho, Wo, st);
    else dx_fewc_launch<CIN, 1>(d, dy, w, dx, Ho, Wo, st);
    count_launch();
    return check_launch("dx_fewc_kernel");
}

int generic_conv_bwd_data(const AetherConvDesc& d, const float* dy, const float* w, float* dx, void* ws, size_t ws_bytes, cudaStream_t st) {
    int Ho, Wo;
    conv_out_hw(d, Ho, Wo);
    // (Few input channels leave a GEMM tile's columns empty.  More than 65535 pixel classes do not fit one grid.)
    if (d.Cin <= 4 && 1LL * d.sH * d.sW <= 65535) {
        switch (d.Cin) {
            case 1: return dx_fewc<1>(d, dy, w, dx, Ho, Wo, st);
            case 2: return dx_fewc<2>(d, dy, w, dx, Ho, Wo, st);
            case 3: return dx_fewc<3>(d, dy, w, dx, Ho, Wo, st);
            default: return dx_fewc<4>(d, dy, w, dx, Ho, Wo, st);
        }
    }
    if (head_shape(d) && (reinterpret_cast<uintptr_t>(dx) & 15u) == 0) return head_dx(d, dy, w, dx, nullptr, st);
    return simt_conv_bwd_data(d, dy, w, dx, ws, ws_bytes, st);
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
