// fp32 convolution on the CUDA cores as tiled implicit GEMMs: every filter size, stride, padding and channel count
// Conv_Layer accepts (CNN/models/CNN_classes_cupy.py:70-154).  It serves what the tensor-core kernels do not take --
// AETHER_MATH_FP32, strided layers, channel counts that are no multiple of 4 -- always in single precision, where the layer is
// too small or has too few channels for conv_split.cu, or no workspace is given.
//
//   forward  y[p][d]  = b[d] + sum_k col[p][k] w[k][d]       M = output pixels, N = Cout, K = taps * Cin
//   dX       dx[q][c] = sum_(tap,d) dy[q - tap][d] w[tap][c][d]   M = input pixels, N = Cin, K = taps * Cout
//   dW       dw[k][d] = sum_p col[p][k] dy[p][d]             M = taps * Cin, N = Cout, K = output pixels, split
//
// Bound by the FMA pipes (74 TFLOP/s): a thread keeps an 8x8 block of sums, so that 64 FMAs share four 16-byte
// shared-memory reads; tiles of 64 or 128 pixels by 16 to 128 channels (SIMT_CONV_TILES, SIMT_DW_TILES) and 16 steps of the
// reduction are staged through registers into
// two shared-memory buffers, the next tile's global loads in flight during the FMAs of the current one.  The reduction
// index walks (filter row, filter column, channel) by mixed-radix steps, so the loop has no division.  A stride s
// splits the input pixels of dX into s*s classes (blockIdx.z) that each see only the taps which reach them; no tap is
// visited that contributes nothing.  Sums run over k in order within a split, splits are added in fixed order.
// Sums are kept in pairs along the output channels for fma.rn.f32x2 (5 % over scalar FMAs: half the issue slots).
// Measured on B200 against one thread per output element: 96 x 28x28 32->64 3x3 fp32, forward + backward, 7.2 -> 0.21 ms;
// 100 x 57x45 48->72 stride 2, 6.3 -> 0.44 ms.  The FMA pipe is 64 % busy in the forward kernel (three warps per scheduler, bound
// by FMA issue; shared memory 50 %, DRAM 2 %); 16 x 8 sums per thread, which halve the warps, are no faster (66 -> 67 us).
#include "common.cuh"
#include "sm100_ptx.cuh"
#include "tc_host.cuh"

namespace aether {

static constexpr int SIMT_BK = 16;

// Asynchronous copies into shared memory; zeros where `ok` is false (nothing is read then).
__device__ __forceinline__ void cp_async16(uint32_t dst, const float* src, bool ok) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Stages of a pipeline whose stage takes `bytes`: three where they fit the 48 KB of static shared memory.
__host__ __device__ constexpr int simt_stages(int bytes) { return 3 * bytes <= 48 * 1024 ? 3 : 2; }

struct SimtGemm {
    const float* in;      // gathered operand: x (forward) or dy (dX), NHWC
    const float* w;       // filter (taps, Cin, Cout)
    const float* bias;    // nullable, N entries (forward)
    float* out;
    int IH, IW, IC;       // extent of `in`
    int N;                // output channels
    int fH, fW;           // filter
    int sH, sW, pH, pW;
    int OH, OW, S;        // extent of `out`
    int Cin, Cout;
    // The tiles behind the first `full` ones (whole rows of tiles) are cut into `parts` pieces of the reduction each, whose
    // sums go to part[class][piece][row behind `row0`][N]; simt_finish_kernel adds them up.
    float* part;
    long long row0, part_rows;
    int full, parts;
    int class0;           // pixel class of blockIdx.z = 0
};

// One side of a tile: BR rows x SIMT_BK reduction steps, four consecutive steps per load.
template <int BR, int THREADS>
struct SimtLoad {
    static constexpr int VPR = SIMT_BK / 4;                 // loads per row
    static constexpr int RPP = THREADS / VPR;               // rows per pass
    static constexpr int L = (BR + RPP - 1) / RPP;          // passes
};

// Position in the reduction (filter row i, filter column j, channel c), advanced without divisions.
struct TapPos {
    int i, j, c;
    __device__ __forceinline__ void init(int k, int C, int nW) {
        const int tap = k / C;
        c = k - tap * C;
        i = tap / nW;
        j = tap - i * nW;
    }
    __device__ __forceinline__ void advance(int dc, int dj, int di, int C, int nW) {
        c += dc; j += dj; i += di;
        if (c >= C) { c -= C; ++j; }
        if (j >= nW) { j -= nW; ++i; }
    }
};

// Thread (tx, ty) of a tile of TX x TY threads: a warp is four threads wide where the tile divides that way, so that the eight
// lanes that a 16-byte shared-memory read serves together share its rows and columns (1-2 %).
template <int TX, int TY>
__device__ __forceinline__ void simt_thread(int tid, int& tx, int& ty) {
    constexpr int WX = (TX % 4 == 0 && TY % 8 == 0) ? 4 : TX, NX = TX / WX;
    if (WX == TX) {
        tx = tid % TX;
        ty = tid / TX;
    } else {
        const int warp = tid >> 5, lane = tid & 31;
        tx = warp % NX * WX + lane % WX;
        ty = warp / NX * (32 / WX) + lane / WX;
    }
}
// CTAs per SM that the register file should hold.
constexpr int simt_ctas(int sums, int threads) { return threads == 256 ? 2 : (sums >= 64 ? 384 : 512) / threads; }

// Two sums at a time (fma.rn.f32x2: the same roundings as two fmaf).
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

template <int BM, int BN, int TM, int TN>
__device__ __forceinline__ void simt_fma_tile(const float (*As)[BM + 4], const float (*Bs)[BN + 4], int ty, int tx,
                                              unsigned long long (&acc)[TM][TN / 2]) {
    constexpr int MH = TM / 4, NH = TN / 4;
#pragma unroll
    for (int k = 0; k < SIMT_BK; ++k) {
        float a[TM];
        unsigned long long b[TN / 2];
#pragma unroll
        for (int q = 0; q < MH; ++q)
            *reinterpret_cast<float4*>(a + 4 * q) = *reinterpret_cast<const float4*>(&As[k][q * (BM / MH) + ty * 4]);
#pragma unroll
        for (int q = 0; q < NH; ++q) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&Bs[k][q * (BN / NH) + tx * 4]);
            b[2 * q] = v.x;
            b[2 * q + 1] = v.y;
        }
#pragma unroll
        for (int m = 0; m < TM; ++m) {
            unsigned long long aa;
            asm("mov.b64 %0, {%1, %1};" : "=l"(aa) : "f"(a[m]));
#pragma unroll
            for (int n = 0; n < TN / 2; ++n) fma2(acc[m][n], aa, b[n]);
        }
    }
}
__device__ __forceinline__ float acc_elem(unsigned long long v, int hi) {
    return __uint_as_float(hi ? (unsigned)(v >> 32) : (unsigned)v);
}

// ---------------------------------------------------------------------------------- forward and dX
// SPLIT: some tiles are cut into pieces (a kernel of its own: the few registers cost the others 2-4 %).
template <int BM, int BN, int TM, int TN, bool DX, bool VEC, bool SPLIT>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), simt_ctas(TM * TN, (BM / TM) * (BN / TN)))
simt_conv_kernel(const SimtGemm g, int n_tiles_n) {
    pdl_wait();
    constexpr int THREADS = (BM / TM) * (BN / TN);
    constexpr int BK = SIMT_BK;
    using LA = SimtLoad<BM, THREADS>;
    using LBT = SimtLoad<BN, THREADS>;                       // DX: filter rows are output channels, steps are contiguous
    constexpr int NB4 = BN / 4;                              // forward: four output channels per load
    constexpr int LBD = (BK * NB4 + THREADS - 1) / THREADS;
    __shared__ __align__(16) float As[2][BK][BM + 4];
    __shared__ __align__(16) float Bs[2][BK][BN + 4];
    const int tid = threadIdx.x;
    int tx, ty;
    simt_thread<BN / TN, BM / TM>(tid, tx, ty);

    // pixel class (dX of a strided layer): rows h = hs + a * sH, taps i = ph + sH * ti
    int ph = 0, pw = 0, nH = g.fH, nW = g.fW, hs = 0, ws = 0, hq = 0, wq = 0, MH = g.OH, MW = g.OW;
    if (DX) {
        const int cls = g.class0 + (int)blockIdx.z;
        ph = cls / g.sW;
        pw = cls - ph * g.sW;
        nH = ph < g.fH ? (g.fH - ph - 1) / g.sH + 1 : 0;
        nW = pw < g.fW ? (g.fW - pw - 1) / g.sW + 1 : 0;
        hs = ((ph - g.pH) % g.sH + g.sH) % g.sH;
        ws = ((pw - g.pW) % g.sW + g.sW) % g.sW;
        hq = (hs + g.pH - ph) / g.sH;                        // exact (hs + pH = ph mod sH) and not negative (ph < sH)
        wq = (ws + g.pW - pw) / g.sW;
        MH = hs < g.OH ? (g.OH - hs - 1) / g.sH + 1 : 0;
        MW = ws < g.OW ? (g.OW - ws - 1) / g.sW + 1 : 0;
    }
    const long long M = 1LL * g.S * MH * MW;
    const int K = nH * nW * g.IC;
    int tile = blockIdx.x, piece = 0, pieces = 1;
    if (SPLIT && tile >= g.full) {
        const int r = tile - g.full;
        pieces = g.parts;
        tile = g.full + r / pieces;
        piece = r % pieces;
    }
    const int nt = tile % n_tiles_n;
    const long long m0 = (long long)(tile / n_tiles_n) * BM;
    const int n0 = nt * BN;
    if (m0 >= M) return;
    const int it0 = SPLIT ? (K + BK - 1) / BK * piece / pieces : 0;

    // rows of the gathered operand this thread loads
    const int kv = tid % LA::VPR, r0 = tid / LA::VPR;
    // (pixel indices are relative to the tile's first sample: 32 bits, widened by the multiplication with the channels)
    const long long s_first = m0 / (1LL * MH * MW);
    const float* in0 = g.in + s_first * g.IH * g.IW * g.IC;
    int a_pix[LA::L], a_h[LA::L], a_w[LA::L];
#pragma unroll
    for (int l = 0; l < LA::L; ++l) {
        const long long m = m0 + r0 + l * LA::RPP;
        if (m < M && r0 + l * LA::RPP < BM) {
            const int wo = (int)(m % MW);
            const long long q = m / MW;
            const int ho = (int)(q % MH);
            const int s = (int)(q / MH - s_first);
            a_h[l] = DX ? ho + hq : ho * g.sH - g.pH;
            a_w[l] = DX ? wo + wq : wo * g.sW - g.pW;
            a_pix[l] = (s * g.IH + a_h[l]) * g.IW + a_w[l];
        } else {
            a_h[l] = -(1 << 28); a_w[l] = 0; a_pix[l] = 0;  // fails every bounds check
        }
    }
    // mixed-radix form of one step of BK
    const int dc = BK % g.IC, dtap = BK / g.IC;
    const int dj = nW > 0 ? dtap % nW : 0, di = nW > 0 ? dtap / nW : 0;
    TapPos pos;
    pos.init(it0 * BK + kv * 4, g.IC, nW > 0 ? nW : 1);
    int k_next = it0 * BK + kv * 4;                          // first reduction step of this thread's next loads
    int kb_next = it0 * BK;                                  // first reduction step of the next tile

    float4 ra[LA::L], rb[DX ? LBT::L : LBD];
    auto load_a4 = [&](const TapPos& t, int l) {
        const int h = DX ? a_h[l] - t.i : a_h[l] + t.i, w = DX ? a_w[l] - t.j : a_w[l] + t.j;
        const int off = t.i * g.IW + t.j;
        return ((unsigned)h < (unsigned)g.IH && (unsigned)w < (unsigned)g.IW) ? in0 + (long long)(DX ? a_pix[l] - off : a_pix[l] + off) * g.IC + t.c
                                                                              : nullptr;
    };
    auto load_tile = [&]() {
        if (VEC) {
            const bool k_ok = k_next < K;
#pragma unroll
            for (int l = 0; l < LA::L; ++l) {
                const float* p = k_ok ? load_a4(pos, l) : nullptr;
                ra[l] = p ? __ldg(reinterpret_cast<const float4*>(p)) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
            if (DX) {
#pragma unroll
                for (int l = 0; l < LBT::L; ++l) {
                    const int n = n0 + r0 + l * LBT::RPP;
                    const float* p = g.w + ((size_t)((ph + pos.i * g.sH) * g.fW + pw + pos.j * g.sW) * g.Cin + n) * g.Cout + pos.c;
                    rb[l] = (k_ok && n < g.N) ? __ldg(reinterpret_cast<const float4*>(p)) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
        } else {
            TapPos t = pos;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const bool k_ok = k_next + e < K;
#pragma unroll
                for (int l = 0; l < LA::L; ++l) {
                    const float* p = k_ok ? load_a4(t, l) : nullptr;
                    reinterpret_cast<float*>(&ra[l])[e] = p ? __ldg(p) : 0.f;
                }
                if (DX) {
#pragma unroll
                    for (int l = 0; l < LBT::L; ++l) {
                        const int n = n0 + r0 + l * LBT::RPP;
                        const float* p = g.w + ((size_t)((ph + t.i * g.sH) * g.fW + pw + t.j * g.sW) * g.Cin + n) * g.Cout + t.c;
                        reinterpret_cast<float*>(&rb[l])[e] = (k_ok && n < g.N) ? __ldg(p) : 0.f;
                    }
                }
                t.advance(1, 0, 0, g.IC, nW);
            }
        }
        if (!DX) {                                           // filter rows k are contiguous in the output channel
#pragma unroll
            for (int l = 0; l < LBD; ++l) {
                const int e = tid + l * THREADS;
                const int kk = e / NB4, n = n0 + (e - kk * NB4) * 4;
                const int k = kb_next + kk;
                rb[l] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (kk < BK && k < K) {
                    const float* p = g.w + (size_t)k * g.Cout + n;
                    if (VEC) {
                        if (n < g.N) rb[l] = __ldg(reinterpret_cast<const float4*>(p));
                    } else {
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (n + q < g.N) reinterpret_cast<float*>(&rb[l])[q] = __ldg(p + q);
                    }
                }
            }
        }
        pos.advance(dc, dj, di, g.IC, nW);
        k_next += BK;
        kb_next += BK;
    };
    auto store_tile = [&](int buf) {
#pragma unroll
        for (int l = 0; l < LA::L; ++l) {
            const int r = r0 + l * LA::RPP;
            if (r < BM) {
                As[buf][kv * 4 + 0][r] = ra[l].x; As[buf][kv * 4 + 1][r] = ra[l].y;
                As[buf][kv * 4 + 2][r] = ra[l].z; As[buf][kv * 4 + 3][r] = ra[l].w;
            }
        }
        if (DX) {
#pragma unroll
            for (int l = 0; l < LBT::L; ++l) {
                const int r = r0 + l * LBT::RPP;
                if (r < BN) {
                    Bs[buf][kv * 4 + 0][r] = rb[l].x; Bs[buf][kv * 4 + 1][r] = rb[l].y;
                    Bs[buf][kv * 4 + 2][r] = rb[l].z; Bs[buf][kv * 4 + 3][r] = rb[l].w;
                }
            }
        } else {
#pragma unroll
            for (int l = 0; l < LBD; ++l) {
                const int e = tid + l * THREADS;
                const int kk = e / NB4;
                if (kk < BK) *reinterpret_cast<float4*>(&Bs[buf][kk][(e - kk * NB4) * 4]) = rb[l];
            }
        }
    };

    unsigned long long acc[TM][TN / 2];
#pragma unroll
    for (int m = 0; m < TM; ++m)
#pragma unroll
        for (int n = 0; n < TN / 2; ++n) acc[m][n] = 0ull;
    const int iters = SPLIT ? (K + BK - 1) / BK * (piece + 1) / pieces - it0 : (K + BK - 1) / BK;
    if (iters > 0) {
        load_tile();
        store_tile(0);
        __syncthreads();
    }
    for (int it = 0; it < iters; ++it) {
        if (it + 1 < iters) load_tile();
        simt_fma_tile<BM, BN, TM, TN>(As[it & 1], Bs[it & 1], ty, tx, acc);
        if (it + 1 < iters) {
            store_tile((it + 1) & 1);
            __syncthreads();
        }
    }

    constexpr int QM = TM / 4, QN = TN / 4;
    const bool vec_out = (g.N & 3) == 0;
    const bool split = SPLIT && pieces > 1;
    const float* bias = DX || split ? nullptr : g.bias;
    float* const out = split ? g.part + (((size_t)g.class0 + blockIdx.z) * pieces + piece) * g.part_rows * g.N : g.out;
#pragma unroll
    for (int qm = 0; qm < QM; ++qm)
#pragma unroll
        for (int mi = 0; mi < 4; ++mi) {
            const long long m = m0 + qm * (BM / QM) + ty * 4 + mi;
            if (m >= M) continue;
            long long pix = split ? m - g.row0 : m;
            if (DX && !split && (g.sH > 1 || g.sW > 1)) {
                const int wo = (int)(m % MW);
                const long long q = m / MW;
                pix = ((q / MH) * g.OH + hs + (q % MH) * g.sH) * g.OW + ws + 1LL * wo * g.sW;
            }
            float* o = out + (size_t)pix * g.N;
#pragma unroll
            for (int qn = 0; qn < QN; ++qn) {
                const int n = n0 + qn * (BN / QN) + tx * 4;
                float v[4];
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    v[e] = acc_elem(acc[qm * 4 + mi][qn * 2 + (e >> 1)], e & 1) + ((!DX && bias != nullptr && n + e < g.N) ? __ldg(bias + n + e) : 0.f);
                if (vec_out) {
                    if (n < g.N) *reinterpret_cast<float4*>(o + n) = make_float4(v[0], v[1], v[2], v[3]);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (n + e < g.N) o[n + e] = v[e];
                }
            }
        }
}

// The rows behind `row0`: the pieces' sums in order, and the bias.  A thread per V channels; four loads in flight.
template <bool DX, int V>
__global__ void __launch_bounds__(256) simt_finish_kernel(const SimtGemm g) {
    pdl_wait();
    int hs = 0, ws = 0, MH = g.OH, MW = g.OW;
    if (DX) {
        const int cls = g.class0 + (int)blockIdx.z, ph = cls / g.sW, pw = cls - ph * g.sW;
        hs = ((ph - g.pH) % g.sH + g.sH) % g.sH;
        ws = ((pw - g.pW) % g.sW + g.sW) % g.sW;
        MH = hs < g.OH ? (g.OH - hs - 1) / g.sH + 1 : 0;
        MW = ws < g.OW ? (g.OW - ws - 1) / g.sW + 1 : 0;
    }
    const long long M = 1LL * g.S * MH * MW;
    const int NV = g.N / V;
    const long long i = 1LL * blockIdx.x * 256 + threadIdx.x;
    const long long row = i / NV, m = g.row0 + row;
    if (row >= g.part_rows || m >= M) return;
    const int n = (int)(i - row * NV) * V;
    const size_t step = (size_t)g.part_rows * g.N;
    const float* p = g.part + ((size_t)g.class0 + blockIdx.z) * g.parts * step + (size_t)row * g.N + n;
    float s[V];
#pragma unroll
    for (int e = 0; e < V; ++e) s[e] = 0.f;
#pragma unroll 4
    for (int q = 0; q < g.parts; ++q) {
        float v[V];
        if constexpr (V == 4) *reinterpret_cast<float4*>(v) = __ldcg(reinterpret_cast<const float4*>(p + q * step));
        else v[0] = __ldcg(p + q * step);
#pragma unroll
        for (int e = 0; e < V; ++e) s[e] += v[e];
    }
    if (!DX && g.bias != nullptr) {
#pragma unroll
        for (int e = 0; e < V; ++e) s[e] += __ldg(g.bias + n + e);
    }
    long long pix = m;
    if (DX && (g.sH > 1 || g.sW > 1)) {
        const int wo = (int)(m % MW);
        const long long q = m / MW;
        pix = ((q / MH) * g.OH + hs + (q % MH) * g.sH) * g.OW + ws + 1LL * wo * g.sW;
    }
    float* o = g.out + (size_t)pix * g.N + n;
    if constexpr (V == 4) *reinterpret_cast<float4*>(o) = make_float4(s[0], s[1], s[2], s[3]);
    else *o = s[0];
}

// ---------------------------------------------------------------------------------- dW, dB
struct SimtDw {
    const float* x;       // nullable: only dB is wanted
    const float* dy;
    float* part;          // [splits][KK + 1][Cout]: row KK holds the split's column sums of dy
    int S, H, W, Cin, Cout, fW, sH, sW, pH, pW, Ho, Wo;
    int KK;               // fH * fW * Cin
    long long P;          // output pixels
    long long per_split;  // a multiple of SIMT_BK
};

// VEC: both operands go straight into shared memory (cp.async, two steps ahead): no staging registers and no stores between the
// FMAs (64 x 32x32 96->96 with the 64 x 64 tile 403 -> 311 us, 96 x 28x28 32->64 75 -> 67 us).  Rows that take four-byte
// loads are staged through registers (457 x 26x26 3->93: 100 us, asynchronously 115), and so are the forward pass and dX: their
// gathered operand is transposed on the way, which four-byte copies do more slowly (dX 76 -> 83 us) and reading it
// untransposed no faster (66 us); they wait for FMA issue (pipe 64 % busy with three warps per scheduler), not for memory.
template <int BM, int BN, int TM, int TN, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), simt_ctas(TM * TN, (BM / TM) * (BN / TN)))
simt_dw_kernel(const SimtDw g, int n_tiles_n) {
    pdl_wait();
    constexpr int THREADS = (BM / TM) * (BN / TN);
    constexpr int BK = SIMT_BK;
    constexpr int MV = BM / 4, NV = BN / 4;                  // loads per pixel
    constexpr int LA = (BK * MV + THREADS - 1) / THREADS, LB = (BK * NV + THREADS - 1) / THREADS;
    static_assert(THREADS % MV == 0 && THREADS >= BN, "a thread keeps its filter entries; one thread per column for dB");
    constexpr int STAGES = simt_stages(BK * (BM + BN + 8) * 4);
    __shared__ __align__(16) float As[STAGES][BK][BM + 4];
    __shared__ __align__(16) float Bs[STAGES][BK][BN + 4];
    const int tid = threadIdx.x;
    int tx, ty;
    simt_thread<BN / TN, BM / TM>(tid, tx, ty);
    const int kt = blockIdx.x / n_tiles_n, nt = blockIdx.x - kt * n_tiles_n;
    const int k0 = kt * BM, n0 = nt * BN;
    const long long p_begin = blockIdx.y * g.per_split;
    const long long p_end = p_begin + g.per_split < g.P ? p_begin + g.per_split : g.P;

    // filter entries of this thread's x loads: four consecutive ones (the same tap when VEC)
    const int mv = tid % MV;
    int ti[4], tj[4], tc[4];
    bool e_ok[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int k = k0 + mv * 4 + e;
        const int tap = k / g.Cin;
        tc[e] = k - tap * g.Cin;
        ti[e] = tap / g.fW;
        tj[e] = tap - ti[e] * g.fW;
        e_ok[e] = g.x != nullptr && k < g.KK;
    }
    // pixels of this thread's x loads, advanced by BK in mixed radix
    const int ds = BK / (g.Ho * g.Wo), drem = BK - ds * g.Ho * g.Wo, dh = drem / g.Wo, dwo = drem - dh * g.Wo;
    // (samples are counted from the split's first one)
    const long long s_first = p_begin / (1LL * g.Ho * g.Wo);
    const float* x0 = g.x != nullptr ? g.x + s_first * g.H * g.W * g.Cin : g.dy;   // (without x nothing is read from it)
    int q_w[LA], q_h[LA], q_s[LA];
#pragma unroll
    for (int l = 0; l < LA; ++l) {
        const long long p = p_begin + tid / MV + l * (THREADS / MV);
        q_w[l] = (int)(p % g.Wo);
        const long long r = p / g.Wo;
        q_h[l] = (int)(r % g.Ho);
        q_s[l] = (int)(r / g.Ho - s_first);
    }
    long long pb = p_begin;
    auto issue = [&](int st) {
#pragma unroll
        for (int l = 0; l < LA; ++l) {
            const int pl = tid / MV + l * (THREADS / MV);
            if (pl < BK) {
                const bool p_ok = pb + pl < p_end;
                const int h0 = q_h[l] * g.sH - g.pH, w0 = q_w[l] * g.sW - g.pW;
                const uint32_t dst = smem_u32(&As[st][pl][mv * 4]);
                const int h = h0 + ti[0], w = w0 + tj[0];
                const bool ok = p_ok && e_ok[0] && (unsigned)h < (unsigned)g.H && (unsigned)w < (unsigned)g.W;
                cp_async16(dst, ok ? x0 + (long long)((q_s[l] * g.H + h) * g.W + w) * g.Cin + tc[0] : g.dy, ok);
            }
            q_w[l] += dwo; q_h[l] += dh; q_s[l] += ds;
            if (q_w[l] >= g.Wo) { q_w[l] -= g.Wo; ++q_h[l]; }
            if (q_h[l] >= g.Ho) { q_h[l] -= g.Ho; ++q_s[l]; }
        }
#pragma unroll
        for (int l = 0; l < LB; ++l) {
            const int e = tid + l * THREADS;
            const int pl = e / NV, n = n0 + (e - pl * NV) * 4;
            if (pl < BK) {
                const float* p = g.dy + (size_t)(pb + pl) * g.Cout + n;
                const uint32_t dst = smem_u32(&Bs[st][pl][(e - pl * NV) * 4]);
                const bool ok = pb + pl < p_end && n < g.Cout;
                cp_async16(dst, ok ? p : g.dy, ok);
            }
        }
        pb += BK;
    };

    float4 ra[LA], rb[LB];
    auto load_tile = [&]() {
#pragma unroll
        for (int l = 0; l < LA; ++l) {
            const int pl = tid / MV + l * (THREADS / MV);
            const bool p_ok = pl < BK && pb + pl < p_end;
            const int h0 = q_h[l] * g.sH - g.pH, w0 = q_w[l] * g.sW - g.pW;
            ra[l] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int h = h0 + ti[e], w = w0 + tj[e];
                if (p_ok && e_ok[e] && (unsigned)h < (unsigned)g.H && (unsigned)w < (unsigned)g.W)
                    reinterpret_cast<float*>(&ra[l])[e] = __ldg(x0 + (long long)((q_s[l] * g.H + h) * g.W + w) * g.Cin + tc[e]);
            }
            q_w[l] += dwo; q_h[l] += dh; q_s[l] += ds;
            if (q_w[l] >= g.Wo) { q_w[l] -= g.Wo; ++q_h[l]; }
            if (q_h[l] >= g.Ho) { q_h[l] -= g.Ho; ++q_s[l]; }
        }
#pragma unroll
        for (int l = 0; l < LB; ++l) {
            const int e = tid + l * THREADS;
            const int pl = e / NV, n = n0 + (e - pl * NV) * 4;
            rb[l] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (pl < BK && pb + pl < p_end) {
                const float* p = g.dy + (size_t)(pb + pl) * g.Cout + n;
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (n + q < g.Cout) reinterpret_cast<float*>(&rb[l])[q] = __ldg(p + q);
            }
        }
        pb += BK;
    };
    auto store_tile = [&](int buf) {
#pragma unroll
        for (int l = 0; l < LA; ++l) {
            const int pl = tid / MV + l * (THREADS / MV);
            if (pl < BK) *reinterpret_cast<float4*>(&As[buf][pl][mv * 4]) = ra[l];
        }
#pragma unroll
        for (int l = 0; l < LB; ++l) {
            const int e = tid + l * THREADS;
            const int pl = e / NV;
            if (pl < BK) *reinterpret_cast<float4*>(&Bs[buf][pl][(e - pl * NV) * 4]) = rb[l];
        }
    };

    unsigned long long acc[TM][TN / 2];
    float bsum = 0.f;
#pragma unroll
    for (int m = 0; m < TM; ++m)
#pragma unroll
        for (int n = 0; n < TN / 2; ++n) acc[m][n] = 0ull;
    const bool sum_dy = kt == 0 && tid < BN;                 // one tile row of the grid adds up dy's columns for dB
    const int iters = p_end > p_begin ? (int)((p_end - p_begin + BK - 1) / BK) : 0;
    auto fma_step = [&](int st) {
        simt_fma_tile<BM, BN, TM, TN>(As[st], Bs[st], ty, tx, acc);
        if (sum_dy) {
#pragma unroll
            for (int k = 0; k < BK; ++k) bsum += Bs[st][k][tid];
        }
    };
    if constexpr (VEC) {
#pragma unroll
        for (int q = 0; q < STAGES - 1; ++q) {
            if (q < iters) issue(q);
            cp_async_commit();
        }
        int st = 0;
        for (int it = 0; it < iters; ++it) {
            cp_async_wait<STAGES - 2>();
            __syncthreads();
            const int nx = st == 0 ? STAGES - 1 : st - 1;
            if (it + STAGES - 1 < iters) issue(nx);
            cp_async_commit();
            fma_step(st);
            st = st + 1 == STAGES ? 0 : st + 1;
        }
    } else {
        if (iters > 0) {
            load_tile();
            store_tile(0);
            __syncthreads();
        }
        for (int it = 0; it < iters; ++it) {
            if (it + 1 < iters) load_tile();
            fma_step(it & 1);
            if (it + 1 < iters) {
                store_tile((it + 1) & 1);
                __syncthreads();
            }
        }
    }

    float* out = g.part + (size_t)blockIdx.y * (g.KK + 1) * g.Cout;
    constexpr int QM = TM / 4, QN = TN / 4;
    const bool vec_out = (g.Cout & 3) == 0;
#pragma unroll
    for (int qm = 0; qm < QM; ++qm)
#pragma unroll
        for (int mi = 0; mi < 4; ++mi) {
            const int k = k0 + qm * (BM / QM) + ty * 4 + mi;
            if (k >= g.KK) continue;
#pragma unroll
            for (int qn = 0; qn < QN; ++qn) {
                const int n = n0 + qn * (BN / QN) + tx * 4;
                float v[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] = acc_elem(acc[qm * 4 + mi][qn * 2 + (e >> 1)], e & 1);
                float* o = out + (size_t)k * g.Cout + n;
                if (vec_out) {
                    if (n < g.Cout) *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (n + e < g.Cout) o[e] = v[e];
                }
            }
        }
    if (sum_dy && n0 + tid < g.Cout) out[(size_t)g.KK * g.Cout + n0 + tid] = bsum;
}

// ---------------------------------------------------------------------------------- host
// An SM takes as many CTAs of a tile at a time as its registers hold (`ctas`) and works at `rate` then (relative; with
// simt_rounds and simt_pick below fitted to the times of all six tiles at fourteen shapes, 6 % off on average).
struct SimtTile { int bm, bn, ctas; double rate; };
static constexpr SimtTile SIMT_CONV_TILES[] = {{128, 128, 2, 1.1},  {128, 64, 3, 1.13},  {64, 64, 6, 1.02},
                                               {128, 32, 4, 0.87}, {128, 16, 4, 0.57}, {64, 32, 4, 0.7}};
static constexpr size_t SIMT_PART_BYTES = 32u << 20;          // most that the pieces of split tiles may take
struct SimtPick {
    int tile, parts;
    long long M, mt, full_mt;                                 // rows, rows of tiles, those of them that are not split
    int classes;
    size_t part_bytes;
};

// Time of the busiest SM in CTAs at full rate when each SM has `per_sm` of them.
static double simt_rounds(long long per_sm, int ctas) {
    const long long rest = per_sm % ctas;
    return (double)(per_sm - rest) + (rest ? rest / (0.4 + 0.6 * rest / ctas) : 0.0);
}

// Tile of the forward pass and dX: the one whose busiest SM is through first.  The tiles behind the last full round of the SMs
// (all of them when they fill no round) may be cut into pieces of the reduction: a small layer leaves SMs without any work
// (8 x 14x14 64->96: 20 + 30 -> 14 + 16 us forward and dX).  A tile costs its steps and four more to start and end (SIMT_STEP_US:
// a step of a 128 x 64 tile of rate 1); pieces must be worth their way through memory (3 TB/s) and the second launch.
static constexpr double SIMT_STEP_US = 0.745;
template <bool DX>
static SimtPick simt_pick(const AetherConvDesc& d, size_t ws_bytes) {
    int Ho, Wo;
    conv_out_hw(d, Ho, Wo);
    SimtPick best{};
    const int N = DX ? d.Cin : d.Cout, sms = num_sms();
    best.classes = DX ? (int)(1LL * d.sH * d.sW < 0x7fffffffLL ? 1LL * d.sH * d.sW : 0x7fffffffLL) : 1;
    best.M = DX ? 1LL * d.S * ceil_div(d.H, d.sH) * ceil_div(d.W, d.sW) : 1LL * d.S * Ho * Wo;    // (pixels of the largest class)
    const double steps = (double)d.fH * d.fW * (DX ? d.Cout : d.Cin) / best.classes / SIMT_BK;
    double best_us = 1e300;
    for (int i = 0; i < (int)(sizeof(SIMT_CONV_TILES) / sizeof(SimtTile)); ++i) {
        const SimtTile& t = SIMT_CONV_TILES[i];
        const long long mt = (best.M + t.bm - 1) / t.bm;
        const int ntn = ceil_div(N, t.bn);
        const double step_us = SIMT_STEP_US * t.bm * t.bn / (128.0 * 64) / t.rate, unit = step_us * (steps + 4.0);
        const long long count = mt * ntn * best.classes, slots = 1LL * t.ctas * sms;
        // (strided dX: its classes have tiles of their own lengths and are split as a whole or not at all)
        const long long rounds = best.classes == 1 ? count / slots : 0, full_mt = rounds * slots / ntn;
        for (int q = 1; q <= 16; ++q) {
            SimtPick p = best;
            p.tile = i;
            p.parts = q;
            p.mt = mt;
            p.full_mt = q == 1 ? mt : full_mt;
            double us;
            if (q == 1) {
                us = unit * simt_rounds((count + sms - 1) / sms, t.ctas);
                p.part_bytes = 0;
            } else {
                const long long rest = (mt - full_mt) * ntn * best.classes * q;
                p.part_bytes = (size_t)best.classes * q * (mt - full_mt) * t.bm * N * sizeof(float);
                if (rest == 0 || steps < 4.0 * q || p.part_bytes > ws_bytes || p.part_bytes > SIMT_PART_BYTES) break;
                us = unit * (double)(rounds * t.ctas) + step_us * (steps / q + 4.0) * simt_rounds((rest + sms - 1) / sms, t.ctas) +
                     3.5 + p.part_bytes * 2 / 3e6;
            }
            if (us < best_us) {
                best_us = us;
                best = p;
            }
        }
    }
    return best;
}

template <int BM, int BN, int TM, int TN, bool DX>
static int launch_simt_conv(SimtGemm g, const SimtPick& p, bool vec, void* ws, cudaStream_t st) {
    const int ntn = ceil_div(g.N, BN);
    const bool split = p.parts > 1;
    g.row0 = p.full_mt * BM;
    g.part_rows = (p.mt - p.full_mt) * BM;
    g.parts = p.parts;
    g.part = static_cast<float*>(ws);
    const long long ctas = (p.full_mt + (p.mt - p.full_mt) * p.parts) * ntn;
    if (ctas > 0x7fffffffLL) return set_error(AE_UNSUPPORTED, "convolution of %lld pixels and %d channels is too large", p.M, g.N);
    g.full = (int)(p.full_mt * ntn);
    constexpr int THREADS = (BM / TM) * (BN / TN), MOST = 65535;       // (classes a grid takes along z)
    const bool v4 = g.N % 4 == 0 && aligned16(g.out) && aligned16(g.part);
    const long long items = g.part_rows * (v4 ? g.N / 4 : g.N);
    for (g.class0 = 0; g.class0 < p.classes; g.class0 += MOST) {
        const unsigned classes = (unsigned)(p.classes - g.class0 < MOST ? p.classes - g.class0 : MOST);
        const dim3 grid((unsigned)ctas, 1, classes);
        if (split) launch(vec ? simt_conv_kernel<BM, BN, TM, TN, DX, true, true> : simt_conv_kernel<BM, BN, TM, TN, DX, false, true>, grid, THREADS, 0, st, g, ntn);
        else launch(vec ? simt_conv_kernel<BM, BN, TM, TN, DX, true, false> : simt_conv_kernel<BM, BN, TM, TN, DX, false, false>, grid, THREADS, 0, st, g, ntn);
        count_launch();
        if (int rc = check_launch("simt_conv_kernel")) return rc;
        if (!split) continue;
        launch(v4 ? simt_finish_kernel<DX, 4> : simt_finish_kernel<DX, 1>, dim3((unsigned)((items + 255) / 256), 1, classes), 256, 0, st, g);
        count_launch();
        if (int rc = check_launch("simt_finish_kernel")) return rc;
    }
    return AE_OK;
}

template <bool DX>
static int simt_conv(const SimtGemm& g, const SimtPick& p, bool vec, void* ws, cudaStream_t st) {
    switch (p.tile) {
        case 0: return launch_simt_conv<128, 128, 8, 8, DX>(g, p, vec, ws, st);
        case 1: return launch_simt_conv<128, 64, 8, 8, DX>(g, p, vec, ws, st);
        case 2: return launch_simt_conv<64, 64, 8, 8, DX>(g, p, vec, ws, st);
        case 3: return launch_simt_conv<128, 32, 8, 4, DX>(g, p, vec, ws, st);
        case 4: return launch_simt_conv<128, 16, 4, 4, DX>(g, p, vec, ws, st);
        default: return launch_simt_conv<64, 32, 4, 4, DX>(g, p, vec, ws, st);
    }
}

// The kernels count the pixels of the gathered operand from a tile's first sample in 32 bits.  How many samples may go
// into one launch for that: all of them, unless the 128 rows of a tile meet samples 2^31 pixels apart (strides of thousands).
static constexpr long long SIMT_MOST_PIXELS = 0x7fffffffLL;
static int simt_samples(const AetherConvDesc& d, bool dx, int Ho, int Wo) {
    const long long pixels = dx ? 1LL * Ho * Wo : 1LL * d.H * d.W;
    const long long rows = dx ? 1LL * (d.H / d.sH) * (d.W / d.sW) : 1LL * Ho * Wo;         // a sample's, of the smallest class
    const long long met = 127 / (rows > 1 ? rows : 1) + 2;
    if (met * pixels <= SIMT_MOST_PIXELS) return d.S;
    const long long n = SIMT_MOST_PIXELS / pixels;
    return (int)(n < d.S ? n : d.S);
}

// `n` samples per launch: f(descriptor, elements of the samples before in its input and in its output).
template <typename F>
static int simt_by_samples(const AetherConvDesc& d, int n, long long in_sample, long long out_sample, F f) {
    if (n < 1) return set_error(AE_UNSUPPORTED, "convolution of %dx%d images: more than 2^31 pixels each", d.H, d.W);
    for (int s = 0; s < d.S; s += n) {
        AetherConvDesc c = d;
        c.S = d.S - s < n ? d.S - s : n;
        if (int rc = f(c, s * in_sample, s * out_sample)) return rc;
    }
    return AE_OK;
}

int simt_conv_fwd(const AetherConvDesc& d, const float* x, const float* w, const float* b, float* y, void* ws, size_t ws_bytes, cudaStream_t st) {
    SimtGemm g{};
    int Ho, Wo;
    conv_out_hw(d, Ho, Wo);
    if (const int n = simt_samples(d, false, Ho, Wo); n < d.S)
        return simt_by_samples(d, n, 1LL * d.H * d.W * d.Cin, 1LL * Ho * Wo * d.Cout, [&](const AetherConvDesc& c, long long in, long long out) {
            return simt_conv_fwd(c, x + in, w, b, y + out, nullptr, 0, st);
        });
    g.in = x; g.w = w; g.bias = b; g.out = y;
    g.IH = d.H; g.IW = d.W; g.IC = d.Cin; g.N = d.Cout;
    g.fH = d.fH; g.fW = d.fW; g.sH = d.sH; g.sW = d.sW; g.pH = d.padH; g.pW = d.padW;
    g.OH = Ho; g.OW = Wo; g.S = d.S; g.Cin = d.Cin; g.Cout = d.Cout;
    const bool vec = d.Cin % 4 == 0 && d.Cout % 4 == 0 && aligned16(x) && aligned16(w) && aligned16(y);
    return simt_conv<false>(g, simt_pick<false>(d, ws ? ws_bytes : 0), vec, ws, st);
}

int simt_conv_bwd_data(const AetherConvDesc& d, const float* dy, const float* w, float* dx, void* ws, size_t ws_bytes, cudaStream_t st) {
    SimtGemm g{};
    int Ho, Wo;
    conv_out_hw(d, Ho, Wo);
    if (const int n = simt_samples(d, true, Ho, Wo); n < d.S)
        return simt_by_samples(d, n, 1LL * Ho * Wo * d.Cout, 1LL * d.H * d.W * d.Cin, [&](const AetherConvDesc& c, long long in, long long out) {
            return simt_conv_bwd_data(c, dy + in, w, dx + out, nullptr, 0, st);
        });
    g.in = dy; g.w = w; g.out = dx;
    g.IH = Ho; g.IW = Wo; g.IC = d.Cout; g.N = d.Cin;
    g.fH = d.fH; g.fW = d.fW; g.sH = d.sH; g.sW = d.sW; g.pH = d.padH; g.pW = d.padW;
    g.OH = d.H; g.OW = d.W; g.S = d.S; g.Cin = d.Cin; g.Cout = d.Cout;
    const bool vec = d.Cin % 4 == 0 && d.Cout % 4 == 0 && aligned16(dy) && aligned16(w) && aligned16(dx);
    return simt_conv<true>(g, simt_pick<true>(d, ws ? ws_bytes : 0), vec, ws, st);
}

// Tile and split of dW: as many splits of the pixels as fill the chip with the tile, each at least eight steps long, and the tile
// whose busiest SM is through first by the estimate of the forward pass and the partials' way through memory (rates measured
// at nine shapes; 128 x 96 is for channel counts that fill two 64-column tiles by three quarters: 64 x 32x32 96->96 307 -> 274 us).
static constexpr SimtTile SIMT_DW_TILES[] = {{128, 128, 2, 1.15}, {128, 64, 3, 1.13}, {64, 64, 6, 1.1},
                                             {64, 32, 4, 0.76},   {32, 64, 4, 0.71},  {128, 96, 2, 0.95}};
struct SimtDwPlan {
    int tile, tiles_k, tiles_n, splits;
    long long per_split;
};
static SimtDwPlan simt_dw_plan(const AetherConvDesc& d) {
    int Ho, Wo;
    conv_out_hw(d, Ho, Wo);
    SimtDwPlan best{};
    const int KK = d.fH * d.fW * d.Cin;
    const long long P = 1LL * d.S * Ho * Wo;
    // (x pixels are counted from a split's first sample in 32 bits: the samples that a split may meet, and so its length)
    const long long met = SIMT_MOST_PIXELS / (1LL * d.H * d.W);
    long long longest = P + SIMT_BK;
    if (met < d.S && met > 2) longest = (met - 2) * Ho * Wo;
    if (longest < SIMT_BK) longest = SIMT_BK;
    double best_us = 1e300;
    for (int i = 0; i < (int)(sizeof(SIMT_DW_TILES) / sizeof(SimtTile)); ++i) {
        const SimtTile& t = SIMT_DW_TILES[i];
        SimtDwPlan p;
        p.tile = i;
        p.tiles_k = ceil_div(KK, t.bm);
        p.tiles_n = ceil_div(d.Cout, t.bn);
        const long long tiles = 1LL * p.tiles_k * p.tiles_n;
        for (int fill = t.ctas; fill >= 1; --fill) {         // CTAs per SM
            long long want = (long long)fill * num_sms() / tiles;
            const long long most = (P + 8 * SIMT_BK - 1) / (8 * SIMT_BK);
            if (want > most) want = most;
            if (want < 1) want = 1;
            if (want > 65535) want = 65535;
            p.per_split = ((P + want - 1) / want + SIMT_BK - 1) / SIMT_BK * SIMT_BK;
            if (p.per_split > longest) p.per_split = longest / SIMT_BK * SIMT_BK;
            p.splits = (int)((P + p.per_split - 1) / p.per_split);
            const double us = simt_rounds((tiles * p.splits + num_sms() - 1) / num_sms(), t.ctas) * SIMT_STEP_US * t.bm * t.bn / (128.0 * 64) /
                                  t.rate * ((double)(p.per_split / SIMT_BK) + 4.0) +
                              (p.splits * 2 + 1) * (double)KK * d.Cout * sizeof(float) / 3e6;
            if (us < best_us) {
                best_us = us;
                best = p;
            }
        }
    }
    return best;
}

size_t simt_conv_workspace_bytes(const AetherConvDesc& d) {
    const size_t entries = (size_t)d.fH * d.fW * d.Cin * d.Cout + d.Cout;
    size_t bytes = align_up((size_t)simt_dw_plan(d).splits * entries * sizeof(float), 1024);
    const size_t fwd = simt_pick<false>(d, SIMT_PART_BYTES).part_bytes, dx = simt_pick<true>(d, SIMT_PART_BYTES).part_bytes;
    bytes = fwd > bytes ? align_up(fwd, 1024) : bytes;
    return dx > bytes ? align_up(dx, 1024) : bytes;
}

template <int BM, int BN, int TM, int TN>
static void launch_simt_dw(const SimtDw& g, const SimtDwPlan& p, bool vec, cudaStream_t st) {
    const dim3 grid((unsigned)(p.tiles_k * p.tiles_n), (unsigned)p.splits);
    constexpr int THREADS = (BM / TM) * (BN / TN);
    if (vec) launch(simt_dw_kernel<BM, BN, TM, TN, true>, grid, THREADS, 0, st, g, p.tiles_n);
    else launch(simt_dw_kernel<BM, BN, TM, TN, false>, grid, THREADS, 0, st, g, p.tiles_n);
    count_launch();
}

int simt_conv_bwd_filter(const AetherConvDesc& d, const float* x, const float* dy, float* dw, float* db, void* ws,
                         size_t ws_bytes, cudaStream_t st) {
    const SimtDwPlan p = simt_dw_plan(d);
    const size_t need = (size_t)p.splits * ((size_t)d.fH * d.fW * d.Cin * d.Cout + d.Cout) * sizeof(float);
    if (!ws || ws_bytes < need) return set_error(AE_BAD_ARG, "conv workspace too small: %zu < %zu", ws_bytes, need);
    SimtDw g{};
    conv_out_hw(d, g.Ho, g.Wo);
    g.x = dw ? x : nullptr; g.dy = dy; g.part = static_cast<float*>(ws);
    g.S = d.S; g.H = d.H; g.W = d.W; g.Cin = d.Cin; g.Cout = d.Cout; g.fW = d.fW;
    g.sH = d.sH; g.sW = d.sW; g.pH = d.padH; g.pW = d.padW;
    g.KK = d.fH * d.fW * d.Cin;
    g.P = 1LL * d.S * g.Ho * g.Wo;
    g.per_split = p.per_split;
    const long long met = p.per_split / (1LL * g.Ho * g.Wo) + 2;
    if ((met < d.S ? met : d.S) * d.H * d.W > SIMT_MOST_PIXELS)
        return set_error(AE_UNSUPPORTED, "filter gradient of %d x %dx%d images: samples too large", d.S, d.H, d.W);
    const bool vec = d.Cin % 4 == 0 && d.Cout % 4 == 0 && aligned16(x) && aligned16(dy);
    switch (p.tile) {
        case 0: launch_simt_dw<128, 128, 8, 8>(g, p, vec, st); break;
        case 1: launch_simt_dw<128, 64, 8, 8>(g, p, vec, st); break;
        case 2: launch_simt_dw<64, 64, 8, 8>(g, p, vec, st); break;
        case 3: launch_simt_dw<64, 32, 4, 4>(g, p, vec, st); break;
        case 4: launch_simt_dw<32, 64, 4, 4>(g, p, vec, st); break;
        default: launch_simt_dw<128, 96, 8, 8>(g, p, vec, st); break;
    }
    int rc = check_launch("simt_dw_kernel");
    if (rc) return rc;
    return smallc_reduce_partials(g.part, p.splits, g.KK, d.Cout, dw, db, st);
}

}  // namespace aether
