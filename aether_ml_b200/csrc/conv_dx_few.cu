// dX of first layers (1..4 input channels), always in single precision:
//
//   dx[s,h,w,c] = sum over taps (i,j) and d of dy[s,ho,wo,d] * w[i,j,c,d] with ho*sH + i - pH == h     (CNN_classes_cupy.py:138-153)
//
// dx_few_tile_kernel takes 3x3 and 5x5 filters at stride 1, dx_few_kernel any other filter or stride.
#include <math.h>
#include <string.h>

#include <type_traits>

#include "common.cuh"
#include "sm100_ptx.cuh"
#include "tc_host.cuh"

namespace aether {

__device__ __forceinline__ void dxf_fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ float dxf_pair_sum(unsigned long long v) { return __uint_as_float((unsigned)v) + __uint_as_float((unsigned)(v >> 32)); }
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

// ---------------------------------------------------------------------------------- stride 1, 3x3 and 5x5
// Bound by the FMA pipes (every value of dy meets CIN * taps filter values), provided that dy comes out of shared memory often enough
// per product and that the copies run beside them.  A lane has a column of R pixels, a warp 32 such columns (TC neighbours in each of 32 / TC strips
// of R rows) and four output channels: its lanes read 16-byte pieces of neighbouring pixels and share the filter's, one
// broadcast each, and a value of dy that has been read meets all filter rows.  The QW warps of the same columns take a chunk of 4 QW channels;
// their sums meet in shared memory at the end of a tile.  Sums are pairs over even and odd channels (fma.rn.f32x2).  Per channel group a
// 3x3 filter on 3 channels takes 432 FMAs (pairs) of a warp and 57 reads.
// A strip's dy with its halo is one TMA box of a chunk's channels (rows of 64 or 128 bytes, swizzled: the 16-byte pieces of eight neighbouring pixels are
// on different banks; pixels outside the image and channels past the last are zeros), copied an item (a chunk of a tile) ahead of the products; blocks
// stay, two per SM.  Rows of dy that are no multiple of 16 bytes are copied by the threads, 4 bytes at a time, into the same places.
// Measured, us, against eight lanes per column of four pixels that read dy and the filter through L1 (dx_few_kernel with the filter's rows in one
// pass): 128 x 32x32 3->32 19.2 / 9.9, 256 x 64x64 3->32 153 / 58, 256 x 32x32 3->128 95 / 62 (25 of FMAs), 100 x 57x52 3->48 5x5 132 / 80, 20 x 64x72
// 3->16 5x5 27 / 14, 200 x 31x31 3->61 87 / 49.  One block per tile, copied by its threads: 11.7, 77, 60, 94, 11, 36; the filter read through L1: 74 for the second.
static constexpr int DXT_THREADS = 256, DXT_STRIPS = 8;      // strips of a tile: at most 4 of a warp x 2 groups of warps

struct DxtParams {
    CUtensorMap tm;                  // dy (Cout, Wo, Ho, S), box of a strip
    CUtensorMap tm_w;                // filter (Cout, taps x Cin), box of a chunk's channels
    const float *dy, *w;
    float* dx;
    int* status;
    int S, H, W, Cout, pH, pW, Ho, Wo;
    int tc_log2, tiles_w, strips;    // columns of a tile, column tiles, strips of an image
    int cols, by_cols;               // columns of dy of a tile, 65536 / cols + 1
    int pixels;                      // of a strip in shared memory: whole swizzle periods
    int chunks, tiles;               // channel chunks, tiles
};

// 16-byte piece q of pixel px (QW pieces per pixel), as TMA places it.
template <int QW>
__device__ __forceinline__ uint32_t dxt_at(uint32_t px, uint32_t q) {
    return QW == 8 ? px * 128u + ((q * 16u) ^ ((px * 16u) & 0x70u)) : px * 64u + ((q * 16u) ^ ((px * 8u) & 0x30u));
}
__host__ __device__ constexpr int dxt_filter_bytes(int rows, int QW) { return (rows * QW * 16 + 1023) / 1024 * 1024; }

// A value of dx next to the left or right end of its row, again, from the arrays: the tile's zeros beside the image times a filter value that is not finite
// are NaN.  (Skipping them in the loop over the filter's columns takes every call longer, 256 x 64x64 3->32 59.3 -> 63.4 us; looking at the results 59.5.)
template <int CIN, int F>
__device__ __noinline__ float dxt_again(const DxtParams& p, int n, int h, int w, int c) {
    float sum = 0.f;
    for (int i = 0; i < F; ++i) {
        const int ho = h + p.pH - i;
        for (int j = 0; j < F; ++j) {
            const int wo = w + p.pW - j;
            if ((unsigned)wo >= (unsigned)p.Wo) continue;
            const bool in = (unsigned)ho < (unsigned)p.Ho;
            const float* g = p.dy + (((size_t)n * p.Ho + (in ? ho : 0)) * p.Wo + wo) * p.Cout;
            const float* k = p.w + (size_t)((i * F + j) * CIN + c) * p.Cout;
            for (int d = 0; d < p.Cout; ++d) sum = fmaf(in ? g[d] : 0.f, k[d], sum);
        }
    }
    return sum;
}

template <int CIN, int F, int QW, int R, bool TMA>
__global__ void __launch_bounds__(DXT_THREADS, 2) dx_few_tile_kernel(const __grid_constant__ DxtParams p) {
    constexpr int ROWS = R + F - 1, PG = 8 / QW, PART = R * 32 * CIN, FILTER = dxt_filter_bytes(F * F * CIN, QW);
    extern __shared__ uint8_t dxt_smem[];
    __shared__ float* out_s[DXT_STRIPS];                     // first pixel of a strip
    __shared__ int rows_s[DXT_STRIPS];                       // its rows
    __shared__ const float* row_s[TMA ? 1 : DXT_STRIPS * ROWS];          // first value of a dy row, null: none
    __shared__ __align__(8) unsigned long long bars[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), q = warp % QW, pg = warp / QW;
    const int G = 32 >> p.tc_log2, TC = 1 << p.tc_log2, strips = PG * G;
    const uint32_t smem = (smem_u32(dxt_smem) + 1023u) & ~1023u;
    uint8_t* gen = dxt_smem + (smem - smem_u32(dxt_smem));
    const uint32_t strip_bytes = (uint32_t)p.pixels * (QW * 16), filter = strips * strip_bytes, stage = filter + FILTER;
    const uint32_t bar0 = smem_u32(bars);
    if (TMA && tid == 0) {
        mbar_init(bar0, 1);
        mbar_init(bar0 + 8, 1);
        mbar_fence_init();
        tma_prefetch_desc(&p.tm);
    }
    pdl_wait();
    if (TMA) __syncthreads();

    // strip k of a tile: image n, first row a0
    auto strip_of = [&](int tile, int k, int& n, int& a0) {
        const unsigned t = (unsigned)(tile / p.tiles_w) * strips + k, i = t / (unsigned)p.strips;
        n = (int)i;
        a0 = (int)(t - i * p.strips) * R;
    };
    auto first_column = [&](int tile) { return (tile % p.tiles_w) << p.tc_log2; };
    // copies of chunk `chunk` of a tile into stage s (TMA: by one thread)
    auto load = [&](int tile, int chunk, uint32_t s) {
        const int col0 = first_column(tile) + p.pW - (F - 1);
        if constexpr (TMA) {
            const uint32_t bar = bar0 + 8 * s;
            int live = 0, n, a0;
            for (int k = 0; k < strips; ++k) {
                strip_of(tile, k, n, a0);
                live += n < p.S;
            }
            mbar_arrive_expect_tx(bar, (uint32_t)live * (ROWS * p.cols * QW * 16) + F * F * CIN * QW * 16);
            tma_load_2d(smem + s * stage + filter, &p.tm_w, bar, chunk * QW * 4, 0);
            for (int k = 0; k < live; ++k) {                 // (strips past the last image come last)
                strip_of(tile, k, n, a0);
                tma_load_4d(smem + s * stage + k * strip_bytes, &p.tm, bar, chunk * QW * 4, col0, a0 + p.pH - (F - 1), n);
            }
        } else {
            const int per_strip = ROWS * p.cols;
            for (int k = 0; k < strips; ++k)
                for (int i = tid; i < per_strip * QW; i += DXT_THREADS) {
                    const int g = i % QW, px = i / QW, row = (px * p.by_cols) >> 16, wo = col0 + px - row * p.cols, d = (chunk * QW + g) * 4;
                    const float* src = row_s[k * ROWS + row];
                    const bool in = src != nullptr && (unsigned)wo < (unsigned)p.Wo;
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const bool ine = in && d + e < p.Cout;
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem + k * strip_bytes + dxt_at<QW>(px, g) + 4 * e),
                                     "l"(ine ? src + (size_t)wo * p.Cout + d + e : p.dy), "r"(ine ? 4 : 0)
                                     : "memory");
                    }
                }
            for (int i = tid; i < F * F * CIN * QW; i += DXT_THREADS) {
                const int g = i % QW, k = i / QW, d = (chunk * QW + g) * 4;
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem + filter + i * 16 + 4 * e),
                                 "l"(p.w + (d + e < p.Cout ? (size_t)k * p.Cout + d + e : 0)), "r"(d + e < p.Cout ? 4 : 0)
                                 : "memory");
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
        }
    };

    if (TMA && tid == 0 && (int)blockIdx.x < p.tiles) load(blockIdx.x, 0, 0);
    const uint32_t px0 = (lane >> p.tc_log2) * p.pixels + (lane & (TC - 1)) + F - 1;         // (whole periods: the swizzle sees the column only)
    uint32_t s = 0, ph = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x) {
        if (tid < strips) {
            int n, a0;
            strip_of(tile, tid, n, a0);
            out_s[tid] = p.dx + (((size_t)n * p.H + a0) * p.W + first_column(tile)) * CIN;
            rows_s[tid] = n < p.S ? min(R, p.H - a0) : 0;
        }
        if (!TMA) {
            for (int i = tid; i < strips * ROWS; i += DXT_THREADS) {
                int n, a0;
                strip_of(tile, i / ROWS, n, a0);
                const int ho = a0 + p.pH - (F - 1) + i % ROWS;
                row_s[i] = n < p.S && (unsigned)ho < (unsigned)p.Ho ? p.dy + ((size_t)n * p.Ho + ho) * p.Wo * p.Cout : nullptr;
            }
            __syncthreads();
        }
        unsigned long long acc[R][CIN];
#pragma unroll
        for (int a = 0; a < R; ++a)
#pragma unroll
            for (int c = 0; c < CIN; ++c) acc[a][c] = 0ull;
        for (int chunk = 0; chunk < p.chunks; ++chunk) {
            if (TMA) {
                // the next item, into the stage that the one before this has left
                const bool more = chunk + 1 < p.chunks;
                const int next = more ? tile : tile + gridDim.x;
                if (tid == 0 && next < p.tiles) load(next, more ? chunk + 1 : 0, s ^ 1u);
                ok = mbar_wait(bar0 + 8 * s, ph, p.status, DS_TIMEOUT_FULL);
            } else {
                load(tile, chunk, 0);
            }
            const int d = (chunk * QW + q) * 4;
            if (d < p.Cout) {
                const uint8_t* dys = gen + s * stage + pg * G * strip_bytes;
                uint32_t px = px0;
                const ulonglong2* wd = reinterpret_cast<const ulonglong2*>(gen + s * stage + filter) + q;
#pragma unroll 1
                for (int j = 0; j < F; ++j, --px, wd += CIN * QW) {
                    ulonglong2 k[F][CIN];
#pragma unroll
                    for (int i = 0; i < F; ++i)
#pragma unroll
                        for (int c = 0; c < CIN; ++c) k[i][c] = wd[(i * F * CIN + c) * QW];
#pragma unroll
                    for (int r = 0; r < ROWS; ++r) {
                        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(dys + dxt_at<QW>(px + r * p.cols, q));
#pragma unroll
                        for (int i = 0; i < F; ++i) {
                            const int a = r - (F - 1) + i;   // the pixel that sees dy row r at filter row i
                            if (a >= 0 && a < R) {
#pragma unroll
                                for (int c = 0; c < CIN; ++c) {
                                    dxf_fma2(acc[a][c], v.x, k[i][c].x);
                                    dxf_fma2(acc[a][c], v.y, k[i][c].y);
                                }
                            }
                        }
                    }
                }
            }
            ok = __syncthreads_and(ok);                      // the stage has been read
            if (chunk + 1 < p.chunks) {
                if (!ok) break;
                s ^= TMA ? 1u : 0u;
                ph ^= s == 0 ? 1u : 0u;
            }
        }
        if (!ok) break;
        // the sums of the tile's warps meet in the stage that has been read last: [warp][pixel of a lane][lane][channel]
        float* red = reinterpret_cast<float*>(gen + s * stage);
#pragma unroll
        for (int a = 0; a < R; ++a)
#pragma unroll
            for (int c = 0; c < CIN; ++c) red[warp * PART + (a * 32 + lane) * CIN + c] = dxf_pair_sum(acc[a][c]);
        __syncthreads();
        const int w0 = first_column(tile);
        bool bad = false;
        for (int e = tid; e < PG * PART; e += DXT_THREADS) {
            const int g = PG > 1 ? e / PART : 0, f = e - g * PART, col = f / CIN, c = f - col * CIN, l = col & 31, a = col >> 5;
            float t[QW];
#pragma unroll
            for (int k = 0; k < QW; ++k) t[k] = red[(g * QW + k) * PART + f];
#pragma unroll
            for (int n = QW / 2; n > 0; n >>= 1)
#pragma unroll
                for (int k = 0; k < n; ++k) t[k] += t[k + n];
            const int strip = g * G + (l >> p.tc_log2), b = l & (TC - 1);
            if (a < rows_s[strip] && w0 + b < p.W) {
                out_s[strip][((size_t)a * p.W + b) * CIN + c] = t[0];
                bad = bad || !isfinite(t[0]);
            }
        }
        for (int e = tid; bad && e < PG * PART; e += DXT_THREADS) {              // (its own values of the loop above)
            const int g = PG > 1 ? e / PART : 0, f = e - g * PART, col = f / CIN, c = f - col * CIN, a = col >> 5;
            const int strip = g * G + ((col & 31) >> p.tc_log2), b = col & (TC - 1), w = w0 + b;
            if (a >= rows_s[strip] || w >= p.W || (w + p.pW >= F - 1 && w + p.pW < p.Wo)) continue;
            float* o = out_s[strip] + ((size_t)a * p.W + b) * CIN + c;
            if (isfinite(*o)) continue;
            int n, a0;
            strip_of(tile, strip, n, a0);
            *o = dxt_again<CIN, F>(p, n, a0 + a, w, c);
        }
        if (TMA) {
            fence_proxy_async_smem();                        // (TMA writes next where the sums were)
            s ^= 1u;
            ph ^= s == 0 ? 1u : 0u;
        }
        __syncthreads();
    }
    if (TMA && !ok && tid == 0) mbar_wait(bar0 + 8 * (s ^ 1u), ph ^ s, p.status, DS_TIMEOUT_FULL);     // (the copy in flight)
}

template <int CIN, int F, int QW, int R, bool TMA>
static int launch_dx_few_tile(DxtParams& p, const AetherConvDesc& d, cudaStream_t st) {
    constexpr int ROWS = R + F - 1, PERIOD = QW == 8 ? 8 : 16;
    const int TC = 1 << p.tc_log2, strips = (8 / QW) * (32 / TC);
    p.cols = TC + F - 1;
    p.by_cols = 65536 / p.cols + 1;
    p.pixels = (ROWS * p.cols + PERIOD - 1) / PERIOD * PERIOD;
    p.tiles_w = ceil_div(d.W, TC);
    p.strips = ceil_div(d.H, R);
    p.tiles = (int)((1LL * d.S * p.strips + strips - 1) / strips * p.tiles_w);
    p.chunks = ceil_div(d.Cout, 4 * QW);
    if (TMA) {
        if (int rc = make_map_nhwc(&p.tm, p.dy, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, d.Cout, p.Wo, p.Ho, d.S, 4 * QW, p.cols, ROWS, 1,
                                   QW == 8 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B))
            return rc;
        if (int rc = make_map_2d(&p.tm_w, p.w, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, d.Cout, F * F * CIN, 4 * QW, F * F * CIN, CU_TENSOR_MAP_SWIZZLE_NONE)) return rc;
    }
    const int smem = 1024 + (TMA ? 2 : 1) * (strips * p.pixels * QW * 16 + dxt_filter_bytes(F * F * CIN, QW));
    static_assert(8 * R * 32 * CIN * 4 <= 32 * 8 / QW * ROWS * QW * 16, "the sums fit a stage");
    static PerDeviceSmem once;
    if (int rc = ensure_dynamic_smem(dx_few_tile_kernel<CIN, F, QW, R, TMA>, smem, once, "dx_few_tile_kernel")) return rc;
    const int most = 2 * num_sms();
    launch(dx_few_tile_kernel<CIN, F, QW, R, TMA>, dim3(p.tiles < most ? p.tiles : most), DXT_THREADS, smem, st, p);
    count_launch();
    return check_launch("dx_few_tile_kernel");
}

// What a tiling costs: rounds of tiles x (products + pixels copied), for 2^tc_log2 columns and R rows.
static double dx_few_cost(const AetherConvDesc& d, int F, int groups, int tc_log2, int R) {
    const int TC = 1 << tc_log2, strips = groups * (32 / TC);
    const double tiles = ceil((double)d.S * ceil_div(d.H, R) / strips) * ceil_div(d.W, TC);
    return ceil(tiles / (2.0 * num_sms())) * (groups * 32 * R + 1.0 * strips * (R + F - 1) * (TC + F - 1));
}

template <int CIN, int F>
static int dx_few_tile(const AetherConvDesc& d, const float* dy, const float* w, float* dx, int Ho, int Wo, cudaStream_t st) {
    constexpr int RL = F == 5 ? 4 : 8;                       // (5x5: the filter column takes the registers)
    // few: four channel groups, two groups of columns.  With 20 channels two such chunks copy less than one of 32 that is a third empty (200 x 28x28
    // 3->20 19.7 / 21.3 us, 53 x 17x17 5.3 / 6.3); with 24 and 28 the sides are even.
    const bool tma = d.Cout % 4 == 0 && aligned16(dy), few = tma && d.Cout <= 20;
    int tc_log2 = 5, R = 4;
    double best = 1e300;
    for (int r = 4; r <= (tma && !few ? RL : 4); r += 4)
        for (int k = 5; k >= 3; --k) {
            const double c = dx_few_cost(d, F, few ? 2 : 1, k, r);
            if (c < best) { best = c; tc_log2 = k; R = r; }
        }
    DxtParams p;
    memset(&p, 0, sizeof(p));
    p.dy = dy; p.w = w; p.dx = dx; p.status = device_status_word();
    p.S = d.S; p.H = d.H; p.W = d.W; p.Cout = d.Cout; p.pH = d.padH; p.pW = d.padW; p.Ho = Ho; p.Wo = Wo;
    p.tc_log2 = tc_log2;
    if (!tma) return launch_dx_few_tile<CIN, F, 8, 4, false>(p, d, st);
    if (few) return launch_dx_few_tile<CIN, F, 4, 4, true>(p, d, st);
    return R == 4 ? launch_dx_few_tile<CIN, F, 8, 4, true>(p, d, st) : launch_dx_few_tile<CIN, F, 8, RL, true>(p, d, st);
}

// ---------------------------------------------------------------------------------- any filter and stride
// Eight lanes share a column of four input pixels and take four output channels each, so a warp's load of dy is four whole 128-byte lines, and one load
// serves FB rows of the filter, which sit in registers: all of a filter of three or five rows at row stride 1, else one at a time.  (us, one at a time / all:
// 128 x 32x32 3->32 3x5 34.4 / 27.4, 5x3 35.0 / 25.5, 3x3 at column stride 2 16.5 / 13.8, 64 x 64x64 3->64 5x1 48.1 / 34.7, 6 x 21x21 1->32 3x5 7.3 / 4.9.)
// Sums are pairs over even and odd channels, the lanes' sums meet in a fixed halving exchange.  A stride splits the input pixels into
// sH * sW classes (blockIdx.z) that each see only the taps that reach them.
static constexpr int DXF_PV = 4;                        // pixels (rows) per thread
static constexpr int DXF_LANES = 8;                     // lanes that share them

template <int CIN, int FB, bool VEC>
__global__ void __launch_bounds__(256, 2) dx_few_kernel(const float* __restrict__ dy, const float* __restrict__ w, float* __restrict__ dx,
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
        for (int c = 0; c < CIN; ++c) f[p][c] = dxf_pair_sum(acc[p][c]);
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

template <int CIN>
static int dx_few(const AetherConvDesc& d, const float* dy, const float* w, float* dx, cudaStream_t st) {
    int Ho, Wo;
    conv_out_hw(d, Ho, Wo);
    // (1x1 filters read each value of dy once, whichever way: 64 x 40x40 3->64 9.0 us through registers, 9.4 through shared memory.  3x3 layers of a few
    // microseconds wait for the host, which takes 0.8 us longer with two tensor maps to encode: 6 x 21x21 1->32, both passes, 16.4 / 17.3; not with more
    // input channels or several chunks of output channels: 5 x 8x8 3->80 11 against 4, one filter row at a time.  Channel counts without tensor maps wait for
    // nothing: 100 x 28x28 1->1 12.9 us through registers, 8.5 so.  Strips and tiles are counted in 32 bits.)
    const bool short_call = CIN == 1 && d.fH == 3 && d.Cout % 4 == 0 && d.Cout <= 32 && 1LL * d.S * Ho * Wo * d.Cout <= 1 << 17;
    if (!short_call && d.sH == 1 && d.sW == 1 && d.fH == d.fW && (d.fH == 3 || d.fH == 5) && 1LL * d.S * d.H * d.W < 0x7fffffffLL)
        return d.fH == 3 ? dx_few_tile<CIN, 3>(d, dy, w, dx, Ho, Wo, st) : dx_few_tile<CIN, 5>(d, dy, w, dx, Ho, Wo, st);
    const bool vec = d.Cout % 4 == 0 && aligned16(dy) && aligned16(w);
    const int MH = ceil_div(d.H, d.sH), MW = ceil_div(d.W, d.sW);            // extent of the largest class
    const long long items = 1LL * d.S * ceil_div(MH, DXF_PV) * MW;
    const dim3 grid((unsigned)((items + 256 / DXF_LANES - 1) / (256 / DXF_LANES)), 1, d.sH * d.sW);
    const auto pick = [&](auto fb) { return vec ? dx_few_kernel<CIN, decltype(fb)::value, true> : dx_few_kernel<CIN, decltype(fb)::value, false>; };
    const int rows = d.sH == 1 && (d.fH == 3 || d.fH == 5) ? d.fH : 1;
    launch(rows == 3 ? pick(std::integral_constant<int, 3>()) : rows == 5 ? pick(std::integral_constant<int, 5>()) : pick(std::integral_constant<int, 1>()), grid, 256, 0, st, dy, w, dx, d.S, d.H, d.W, d.Cout, d.fH, d.fW, d.sH, d.sW,
           d.padH, d.padW, Ho, Wo);
    count_launch();
    return check_launch("dx_few_kernel");
}

int dx_few_conv_bwd_data(const AetherConvDesc& d, const float* dy, const float* w, float* dx, cudaStream_t st) {
    switch (d.Cin) {
        case 1: return dx_few<1>(d, dy, w, dx, st);
        case 2: return dx_few<2>(d, dy, w, dx, st);
        case 3: return dx_few<3>(d, dy, w, dx, st);
        default: return dx_few<4>(d, dy, w, dx, st);
    }
}

}  // namespace aether
