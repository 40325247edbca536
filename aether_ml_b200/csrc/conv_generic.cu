// Single-precision convolution (CNN/models/CNN_classes_cupy.py:70-154) for the shapes the tensor-core kernels do not take:
// classifier heads (pointwise layers with few outputs per pixel) have kernels of their own here, the dX of first layers (1 to 4 input channels)
// has conv_dx_few.cu, everything else goes to the tiled implicit GEMMs of conv_simt.cu.
#include "common.cuh"
#include "tc_host.cuh"

namespace aether {

// Pointwise layers with very few outputs per pixel (a classifier head: Dense 1024 -> 10 is a 1x1 convolution with
// Cout = 10): with one thread per output element a batch of 512 rows is 5120 threads walking 1024 channels each.
// Here a warp takes a row: the lanes split the channels (float4 loads of x, the row is read once), keep Cout partial
// sums each and combine them with shuffles in a fixed order.
// The filter is kept transposed in shared memory, wT[d][Cin], so a lane's four channels of output d are one 16-byte
// shared-memory read (4 * Cout scalar global loads per four channels before).  Its 16-byte loads are all in flight before the first
// store: with scalar ones in a loop of their own the copy was a third of a small layer's time.
// (rows of Cin + 4 floats: with Cin a multiple of 32 the outputs of one channel would all fall on one bank)
__device__ __forceinline__ void head_load_filter_T(const float* __restrict__ w, float* wT, int Cin, int Cout) {
    constexpr int U = 4;
    const int n4 = (Cin * Cout) >> 2;
    for (int i0 = threadIdx.x; i0 < n4; i0 += U * blockDim.x) {
        float4 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (i0 + u * (int)blockDim.x < n4) v[u] = __ldg(reinterpret_cast<const float4*>(w) + i0 + u * (int)blockDim.x);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = i0 + u * (int)blockDim.x;
            if (i >= n4) break;
            int c = (int)(4u * (unsigned)i / (unsigned)Cout), d = 4 * i - c * Cout;
            const float e[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                wT[d * (Cin + 4) + c] = e[k];
                if (++d == Cout) { d = 0; ++c; }
            }
        }
    }
    __syncthreads();
}

// Bound by latency: a batch of 128 rows of 256 channels is 16 blocks and one row per warp.  The first row is requested before the
// filter is copied, and the lanes' sums of 16 outputs meet in four halving exchanges (the lane's output is lane / 2) and one that
// adds: 16 shuffles, in the order of the 80 that a butterfly per output takes.  With its softmax, as
// a train of launches, before / after: 128 x 256->10 4.9 / 3.5 us, 1024 x 1024->10 14.9 / 9.9, 4096 x 1024->10 23.0 / 18.5.
template <int MAXD>
__global__ void __launch_bounds__(256) gen_fwd_pointwise_few_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                                    const float* __restrict__ b, float* __restrict__ y,
                                                                    long long rows, int Cin, int Cout, float* __restrict__ prob) {
    static_assert(MAXD == 16, "the halving exchange below");
    pdl_wait();
    extern __shared__ __align__(16) float head_wT[];
    const int lane = threadIdx.x & 31, out = lane >> 1;
    const long long warp0 = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    const int C4 = Cin >> 2;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 next[2];                                          // the next row's first channels, requested a row ahead
#pragma unroll
    for (int u = 0; u < 2; ++u)
        next[u] = warp0 < rows && lane + 32 * u < C4 ? reinterpret_cast<const float4*>(x + (size_t)warp0 * Cin)[lane + 32 * u] : zero;
    const float bias = b != nullptr && out < Cout ? b[out] : 0.f;
    head_load_filter_T(w, head_wT, Cin, Cout);
    for (long long row = warp0; row < rows; row += nwarps) {
        float acc[MAXD];
#pragma unroll
        for (int d = 0; d < MAXD; ++d) acc[d] = 0.f;
        const float4* xr = reinterpret_cast<const float4*>(x + (size_t)row * Cin);
        const float4 v0 = next[0], v1 = next[1];
#pragma unroll
        for (int u = 0; u < 2; ++u)
            next[u] = row + nwarps < rows && lane + 32 * u < C4 ? reinterpret_cast<const float4*>(x + (size_t)(row + nwarps) * Cin)[lane + 32 * u] : zero;
        for (int c4 = lane; c4 < C4; c4 += 32) {
            const float4 v = c4 < 32 ? v0 : c4 < 64 ? v1 : xr[c4];
#pragma unroll
            for (int d = 0; d < MAXD; ++d) {
                if (d < Cout) {
                    const float4 k = *reinterpret_cast<const float4*>(head_wT + d * (Cin + 4) + 4 * c4);
                    acc[d] = fmaf(v.x, k.x, fmaf(v.y, k.y, fmaf(v.z, k.z, fmaf(v.w, k.w, acc[d]))));
                }
            }
        }
#pragma unroll
        for (int n = MAXD / 2; n > 0; n >>= 1) {             // partner 2 n lanes on: each keeps n of the 2 n outputs
            const bool hi = lane & (2 * n);
#pragma unroll
            for (int d = 0; d < n; ++d) {
                const float give = hi ? acc[d] : acc[d + n], keep = hi ? acc[d + n] : acc[d];
                acc[d] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * n);
            }
        }
        const float sum_x = acc[0] + __shfl_xor_sync(0xffffffffu, acc[0], 1);
        float z = -INFINITY;
        if (out < Cout) {
            z = sum_x + bias;
            if (!(lane & 1)) y[(size_t)row * Cout + out] = z;
        }
        if (prob != nullptr) {                               // the softmax behind the head, as softmax_cce_kernel computes it
            float mx = z;
#pragma unroll
            for (int o = 16; o > 1; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const float e = out < Cout ? expf(z - mx) : 0.f;
            float sum = e;
#pragma unroll
            for (int o = 16; o > 1; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            if (out < Cout && !(lane & 1)) prob[(size_t)row * Cout + out] = e / sum;
        }
    }
}

// ---------------------------------------------------------------------------------- classifier heads, backward
// All of a head's backward pass in one launch: blocks for dW (16 channels each, the first adds dB up), blocks for dX; each is a few round trips
// to L2 long, and one behind the other they were three launches.  With the loss gradient,
// three launches / one: 128 x 256->10 10.4 / 3.2 us, 512 x 512 15.8 / 6.1, 1024 x 1024 25.4 / 12.7, 4096 x 1024 (three launches here, too: labels
// are requested a row ahead) 55.9 / 52.6.  Above HEAD_DW_ROWS rows dW and dB are sums of parts
// (head_dw_partial_kernel below).
//
// dx[p][c] = sum_d dy[p][d] * w[c][d]: a block is row lanes x four-channel groups; the filter is read transposed from shared memory, the
// row of dy is the same address for every thread of a row.  dw[c][d] = sum_p x[p][c] * dy[p][d]: a thread keeps four channels x Cout
// sums over every 64th row (x read once, in 64-byte pieces; dy from shared memory), the sums meet in halving exchanges, then over the warps.
// CCE: dy is not there yet -- it is the combined softmax / cross-entropy gradient (prob - y_smooth) / rows, which is computed
// from the probabilities and the labels of the row (as softmax_cce_kernel does) wherever it is read, and written to dz by the dX blocks.
struct HeadCce {
    const float* prob;
    const int* labels;             // one of the three
    const long long* labels64;
    const float* targets;
    float* dz;
    float smooth, inv_rows;
};
struct HeadBwd {
    const float *x, *dy, *w;
    float *dx, *dw, *db;           // each nullable
    long long rows;
    int Cin, Cout;
    int dw_blocks;                 // the first blocks of the grid (the first of them: dB, too); the rest are dX's
    int lanes, groups;             // dX: rows of a block, threads of a row
    HeadCce cce;
};
static constexpr int HEAD_DW_CH = 16, HEAD_DW_CHUNK = 256, HEAD_DZ_LD = 20;      // (rows of 20 floats: eight rows' reads on 32 banks)
static constexpr int HEAD_DW_SMEM = (HEAD_DW_CHUNK * HEAD_DZ_LD + 8 * 16 * HEAD_DW_CH) * (int)sizeof(float);

__device__ __forceinline__ int head_label(const HeadCce& cce, long long row) {
    return cce.labels ? cce.labels[row] : cce.labels64 ? (int)cce.labels64[row] : -1;
}
// dy at (row, d) from what `v` holds: dy itself or the probability.
template <bool CCE>
__device__ __forceinline__ float head_dy(const HeadCce& cce, float v, long long row, int d, int Cout, int label) {
    if (!CCE) return v;
    const float onehot = cce.targets ? cce.targets[(size_t)row * Cout + d] : (d == label ? 1.f : 0.f);
    const float tb = onehot * (1.f - cce.smooth) + cce.smooth / Cout;
    return (v - tb) * cce.inv_rows;
}

template <int MAXD, bool CCE>
__device__ __forceinline__ void head_dx_block(const HeadBwd& p, int block, int blocks, float* wT) {
    head_load_filter_T(p.w, wT, p.Cin, p.Cout);
    const int C4 = p.Cin >> 2;
    const int rl = (int)threadIdx.x / p.groups, cl = (int)threadIdx.x - rl * p.groups;
    if (rl >= p.lanes) return;
    const float* src = CCE ? p.cce.prob : p.dy;
    const long long row0 = (long long)block * p.lanes + rl, step = (long long)blocks * p.lanes;
    float gn[MAXD];                                     // the next row's dy values and label, requested one row ahead
    int next_label = CCE && row0 < p.rows ? head_label(p.cce, row0) : 0;
#pragma unroll
    for (int d = 0; d < MAXD; ++d) gn[d] = (d < p.Cout && row0 < p.rows) ? __ldg(src + (size_t)row0 * p.Cout + d) : 0.f;
    for (long long row = row0; row < p.rows; row += step) {
        float g[MAXD];
        const long long nrow = row + step;
        const int label = next_label;
        if (CCE && nrow < p.rows) next_label = head_label(p.cce, nrow);
#pragma unroll
        for (int d = 0; d < MAXD; ++d) {
            g[d] = gn[d];
            gn[d] = (d < p.Cout && nrow < p.rows) ? __ldg(src + (size_t)nrow * p.Cout + d) : 0.f;
        }
        if (CCE) {
#pragma unroll
            for (int d = 0; d < MAXD; ++d) {
                if (d < p.Cout) {
                    g[d] = head_dy<CCE>(p.cce, g[d], row, d, p.Cout, label);
                    if (cl == d) p.cce.dz[(size_t)row * p.Cout + d] = g[d];
                }
            }
        }
        float4* out = reinterpret_cast<float4*>(p.dx + (size_t)row * p.Cin);
        for (int c4 = cl; c4 < C4; c4 += p.groups) {
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int d = 0; d < MAXD; ++d) {
                if (d < p.Cout) {
                    const float4 k = *reinterpret_cast<const float4*>(wT + d * (p.Cin + 4) + 4 * c4);
                    a.x = fmaf(g[d], k.x, a.x); a.y = fmaf(g[d], k.y, a.y); a.z = fmaf(g[d], k.z, a.z); a.w = fmaf(g[d], k.w, a.w);
                }
            }
            out[c4] = a;
        }
    }
}

template <int MAXD, bool CCE>
__device__ __forceinline__ void head_dw_block(const HeadBwd& p, int block, float* smem) {
    static_assert(MAXD == 16, "the halving exchange below");
    float* dz_s = smem;
    float* red = smem + HEAD_DW_CHUNK * HEAD_DZ_LD;     // [warp][output][channel]
    const int lane = threadIdx.x & 31, cg = threadIdx.x & 3, rl = threadIdx.x >> 2;
    const int C4 = p.Cin >> 2, c4 = block * (HEAD_DW_CH / 4) + cg, rows = (int)p.rows;
    const float* src = CCE ? p.cce.prob : p.dy;
    float4 acc[MAXD];
#pragma unroll
    for (int d = 0; d < MAXD; ++d) acc[d] = make_float4(0.f, 0.f, 0.f, 0.f);
    float sdy = 0.f;                                    // block 0: column sums of dy, output threadIdx.x & 15, every 16th row
    float4 v[HEAD_DW_CHUNK / 64];                       // this chunk's x, and dy of the thread's own row: requested a chunk ahead
    float g[MAXD];
    int label = 0;
    auto request = [&](int r0) {
#pragma unroll
        for (int u = 0; u < HEAD_DW_CHUNK / 64; ++u) {
            const int r = r0 + u * 64 + rl;
            v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r < rows && c4 < C4) v[u] = __ldg(reinterpret_cast<const float4*>(p.x) + (size_t)r * C4 + c4);
        }
        const int r = r0 + (int)threadIdx.x;
        if (r < rows) {
#pragma unroll
            for (int d = 0; d < MAXD; ++d)
                if (d < p.Cout) g[d] = __ldg(src + (size_t)r * p.Cout + d);
            if (CCE) label = head_label(p.cce, r);
        }
    };
    request(0);
    for (int r0 = 0; r0 < rows; r0 += HEAD_DW_CHUNK) {
        if (r0 > 0) __syncthreads();
        if (r0 + (int)threadIdx.x < rows) {
#pragma unroll
            for (int d = 0; d < MAXD; ++d)
                if (d < p.Cout) dz_s[threadIdx.x * HEAD_DZ_LD + d] = head_dy<CCE>(p.cce, g[d], r0 + (int)threadIdx.x, d, p.Cout, label);
        }
        float4 xv[HEAD_DW_CHUNK / 64];
#pragma unroll
        for (int u = 0; u < HEAD_DW_CHUNK / 64; ++u) xv[u] = v[u];
        if (r0 + HEAD_DW_CHUNK < rows) request(r0 + HEAD_DW_CHUNK);
        __syncthreads();
#pragma unroll
        for (int u = 0; u < HEAD_DW_CHUNK / 64; ++u) {
            if (r0 + u * 64 + rl >= rows) continue;
            const float4* gr = reinterpret_cast<const float4*>(dz_s + (u * 64 + rl) * HEAD_DZ_LD);
#pragma unroll
            for (int q = 0; q < MAXD / 4; ++q) {
                if (4 * q >= p.Cout) break;
                const float4 g4 = gr[q];                // (entries from Cout on are read and not used)
                const float gk[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (4 * q + k < p.Cout) {
                        float4& a = acc[4 * q + k];
                        a.x = fmaf(xv[u].x, gk[k], a.x); a.y = fmaf(xv[u].y, gk[k], a.y);
                        a.z = fmaf(xv[u].z, gk[k], a.z); a.w = fmaf(xv[u].w, gk[k], a.w);
                    }
                }
            }
        }
        if (block == 0 && p.db != nullptr && (threadIdx.x & 15) < p.Cout) {
            const int n = rows - r0 < HEAD_DW_CHUNK ? rows - r0 : HEAD_DW_CHUNK;
            float t[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int l = 0; l < HEAD_DW_CHUNK / 16; ++l) {
                const int r = ((int)threadIdx.x >> 4) + 16 * l;
                if (r < n) t[l & 3] += dz_s[r * HEAD_DZ_LD + (threadIdx.x & 15)];
            }
            sdy += (t[0] + t[1]) + (t[2] + t[3]);
        }
    }
    // A warp's eight rows: partner 2 n lanes on, each keeps n of the 2 n outputs.
#pragma unroll
    for (int n = MAXD / 2; n > 1; n >>= 1) {
        const bool hi = lane & (2 * n);
#pragma unroll
        for (int d = 0; d < n; ++d) {
            const float4 give = hi ? acc[d] : acc[d + n], keep = hi ? acc[d + n] : acc[d];
            acc[d].x = keep.x + __shfl_xor_sync(0xffffffffu, give.x, 2 * n);
            acc[d].y = keep.y + __shfl_xor_sync(0xffffffffu, give.y, 2 * n);
            acc[d].z = keep.z + __shfl_xor_sync(0xffffffffu, give.z, 2 * n);
            acc[d].w = keep.w + __shfl_xor_sync(0xffffffffu, give.w, 2 * n);
        }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k)
        *reinterpret_cast<float4*>(red + ((threadIdx.x >> 5) * MAXD + (lane >> 2) * 2 + k) * HEAD_DW_CH + cg * 4) = acc[k];
    __syncthreads();
    const int c = (int)(threadIdx.x / (unsigned)p.Cout), d = (int)threadIdx.x - c * p.Cout;
    if (p.dw != nullptr && c < HEAD_DW_CH && block * HEAD_DW_CH + c < p.Cin) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) s += red[(w * MAXD + d) * HEAD_DW_CH + c];
        p.dw[(size_t)(block * HEAD_DW_CH + c) * p.Cout + d] = s;
    }
    if (block == 0 && p.db != nullptr) {
        __syncthreads();
        red[threadIdx.x] = sdy;
        __syncthreads();
        if (threadIdx.x < p.Cout) {
            float t[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int l = 0; l < 16; ++l) t[l & 3] += red[l * 16 + threadIdx.x];
            p.db[threadIdx.x] = (t[0] + t[1]) + (t[2] + t[3]);
        }
    }
}

template <int MAXD, bool CCE>
__global__ void __launch_bounds__(256, 2) head_bwd_kernel(const HeadBwd p) {
    pdl_wait();
    extern __shared__ __align__(16) float head_smem[];
    const int b = blockIdx.x;
    if (b < p.dw_blocks) head_dw_block<MAXD, CCE>(p, b, head_smem);
    else head_dx_block<MAXD, CCE>(p, b - p.dw_blocks, gridDim.x - p.dw_blocks, head_smem);
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

int generic_conv_bwd_data(const AetherConvDesc& d, const float* dy, const float* w, float* dx, void* ws, size_t ws_bytes, cudaStream_t st) {
    // (Few input channels leave a GEMM tile's columns empty.  More than 65535 pixel classes do not fit one grid.)
    if (d.Cin <= 4 && 1LL * d.sH * d.sW <= 65535) return dx_few_conv_bwd_data(d, dy, w, dx, st);
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

// Most rows whose dW comes out of one launch: a thread's sum is over every 64th row, 16 of them here, as long as the parts' below.  One
// launch is faster for more rows, too (2048 x 256->10 18.8 us against 21.1, 4096 x 1024->10 41.7 against 52.6), but from there on its longer
// sums are the less accurate ones (dW at 4096 rows 1.30e-7 off float64 against 1.14e-7; at 1024 1.00e-7 against 1.05e-7).
static constexpr int HEAD_DW_ROWS = 1024;

static int head_bwd(const AetherConvDesc& d, const float* x, const float* dy, const float* w, float* dx, float* dw, float* db, void* ws,
                    size_t ws_bytes, const HeadCce* cce, cudaStream_t st) {
    const bool sums = dw != nullptr || db != nullptr;
    if (sums && (!ws || ws_bytes < generic_conv_workspace_bytes(d)))
        return set_error(AE_BAD_ARG, "conv workspace too small: %zu < %zu", ws_bytes, generic_conv_workspace_bytes(d));
    const int C4 = d.Cin / 4;
    HeadBwd p = {};
    p.x = x; p.dy = dy; p.w = w; p.dx = dx; p.dw = dw; p.db = db;
    p.rows = 1LL * d.S * d.H * d.W;
    p.Cin = d.Cin;
    p.Cout = d.Cout;
    if (cce) p.cce = *cce;
    const bool parted = p.rows > HEAD_DW_ROWS;
    p.dw_blocks = !sums || parted ? 0 : dw ? ceil_div(d.Cin, HEAD_DW_CH) : 1;
    p.groups = C4 < 256 ? C4 : 256;
    p.lanes = 256 / p.groups;
    long long dx_blocks = 0;
    if (dx) {
        dx_blocks = (p.rows + p.lanes - 1) / p.lanes;
        // What is resident at once, for every block copies the filter.
        const long long most = p.dw_blocks < num_sms() ? 2LL * num_sms() - p.dw_blocks : num_sms();
        if (dx_blocks > most) dx_blocks = most;
    }
    if (const int grid = p.dw_blocks + (int)dx_blocks) {
        static PerDeviceSmem configured[2];
        const auto kernel = cce ? head_bwd_kernel<16, true> : head_bwd_kernel<16, false>;
        if (int rc = ensure_dynamic_smem(kernel, 96 * 1024, configured[cce ? 1 : 0], "head backward")) return rc;
        const int filter = dx ? (d.Cin + 4) * d.Cout * (int)sizeof(float) : 0, tile = p.dw_blocks ? HEAD_DW_SMEM : 0;
        launch(kernel, grid, 256, filter > tile ? filter : tile, st, p);
        count_launch();
        if (int rc = check_launch("head_bwd_kernel")) return rc;
    }
    if (!sums || !parted) return AE_OK;
    const int parts = head_dw_parts(d);
    int lanes = 1;                                       // row lanes per block: as many as whole channel rows fit 256 threads
    while (lanes * 2 <= parts && C4 * lanes * 2 <= 256) lanes *= 2;
    const int groups = 256 / lanes;
    float* part = static_cast<float*>(ws);
    launch(head_dw_partial_kernel<16>, dim3(ceil_div(parts, lanes), ceil_div(C4, groups)), 256, 0, st, x, cce ? cce->dz : dy, part, p.rows, d.Cin,
           d.Cout, lanes, parts);
    count_launch();
    if (int rc = check_launch("head_dw_partial_kernel")) return rc;
    launch(head_dw_reduce_kernel, ceil_div((d.Cin + 1) * d.Cout, 32), 256, 0, st, part, parts, d.Cin, d.Cout, dw, db);
    count_launch();
    return check_launch("head_dw_reduce_kernel");
}

int generic_head_bwd(const AetherConvDesc& d, const float* x, const float* dy, const float* w, float* dx, float* dw, float* db, void* ws,
                     size_t ws_bytes, cudaStream_t st) {
    return head_bwd(d, x, dy, w, dx, dw, db, ws, ws_bytes, nullptr, st);
}
int generic_head_cce_bwd(const AetherConvDesc& d, const float* prob, const int* labels, const long long* labels64, const float* targets,
                         float smooth, const float* x, const float* w, float* dz, float* dx, float* dw, float* db, void* ws, size_t ws_bytes,
                         cudaStream_t st) {
    const HeadCce cce = {prob, labels, labels64, targets, dz, smooth, 1.f / (float)(1LL * d.S * d.H * d.W)};
    return head_bwd(d, x, nullptr, w, dx, dw, db, ws, ws_bytes, &cce, st);
}

}  // namespace aether
