// fp32 convolution on the CUDA cores as tiled implicit GEMMs: every filter size, stride, padding and channel count
// Conv_Layer accepts (CNN/models/CNN_classes_cupy.py:70-154).  It serves what the tensor-core kernels do not take --
// AETHER_MATH_FP32, strided layers, channel counts that are no multiple of 4 -- always in single precision.
//
//   forward  y[p][d]  = b[d] + sum_k col[p][k] w[k][d]       M = output pixels, N = Cout, K = taps * Cin
//   dX       dx[q][c] = sum_(tap,d) dy[q - tap][d] w[tap][c][d]   M = input pixels, N = Cin, K = taps * Cout
//   dW       dw[k][d] = sum_p col[p][k] dy[p][d]             M = taps * Cin, N = Cout, K = output pixels, split
//
// Bound by the FMA pipes (74 TFLOP/s): a thread keeps an 8x8 block of sums, so that 64 FMAs share four 16-byte
// shared-memory reads; tiles of 128 x {128, 64, 32, 16} and 16 steps of the reduction are staged through registers into
// two shared-memory buffers, the next tile's global loads in flight during the FMAs of the current one.  The reduction
// index walks (filter row, filter column, channel) by mixed-radix steps, so the loop has no division.  A stride s
// splits the input pixels of dX into s*s classes (blockIdx.z) that each see only the taps which reach them; no tap is
// visited that contributes nothing.  Sums run over k in order within a split, splits are added in fixed order.
// Sums are kept in pairs along the output channels for fma.rn.f32x2 (5 % over scalar FMAs: half the issue slots).
// Measured on B200 against one thread per output element: 96 x 28x28 32->64 3x3 fp32, forward + backward, 7.2 -> 0.22 ms
// (43 TFLOP/s, 50 to 63 where the tiles fill whole rounds of the SMs); 100 x 57x45 48->72 stride 2, 6.3 -> 0.46 ms.
#include "common.cuh"
#include "tc_host.cuh"

namespace aether {

static constexpr int SIMT_BK = 16;

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
template <int BM, int BN, int TM, int TN, bool DX, bool VEC>
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
        ph = blockIdx.z / g.sW;
        pw = blockIdx.z - ph * g.sW;
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
    const int nt = blockIdx.x % n_tiles_n;
    const long long m0 = (long long)(blockIdx.x / n_tiles_n) * BM;
    const int n0 = nt * BN;
    if (m0 >= M) return;

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
    pos.init(kv * 4, g.IC, nW > 0 ? nW : 1);
    int k_next = kv * 4;                                     // first reduction step of this thread's next loads
    int kb_next = 0;                                         // first reduction step of the next tile

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
    const int iters = (K + BK - 1) / BK;
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
#pragma unroll
    for (int qm = 0; qm < QM; ++qm)
#pragma unroll
        for (int mi = 0; mi < 4; ++mi) {
            const long long m = m0 + qm * (BM / QM) + ty * 4 + mi;
            if (m >= M) continue;
            long long pix = m;
            if (DX && (g.sH > 1 || g.sW > 1)) {
                const int wo = (int)(m % MW);
                const long long q = m / MW;
                pix = ((q / MH) * g.OH + hs + (q % MH) * g.sH) * g.OW + ws + 1LL * wo * g.sW;
            }
            float* o = g.out + (size_t)pix * g.N;
#pragma unroll
            for (int qn = 0; qn < QN; ++qn) {
                const int n = n0 + qn * (BN / QN) + tx * 4;
                float v[4];
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    v[e] = acc_elem(acc[qm * 4 + mi][qn * 2 + (e >> 1)], e & 1) + ((!DX && g.bias != nullptr && n + e < g.N) ? __ldg(g.bias + n + e) : 0.f);
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

template <int BM, int BN, int TM, int TN, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), simt_ctas(TM * TN, (BM / TM) * (BN / TN)))
simt_dw_kernel(const SimtDw g, int n_tiles_n) {
    pdl_wait();
    constexpr int THREADS = (BM / TM) * (BN / TN);
    constexpr int BK = SIMT_BK;
    constexpr int MV = BM / 4, NV = BN / 4;                  // loads per pixel
    constexpr int LA = (BK * MV + THREADS - 1) / THREADS, LB = (BK * NV + THREADS - 1) / THREADS;
    static_assert(THREADS % MV == 0 && THREADS >= BN, "a thread keeps its filter entries; one thread per column for dB");
    __shared__ __align__(16) float As[2][BK][BM + 4];
    __shared__ __align__(16) float Bs[2][BK][BN + 4];
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
    const float* x0 = g.x + (g.x != nullptr ? s_first * g.H * g.W * g.Cin : 0);
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
    float4 ra[LA], rb[LB];
    auto load_tile = [&]() {
#pragma unroll
        for (int l = 0; l < LA; ++l) {
            const int pl = tid / MV + l * (THREADS / MV);
            const bool p_ok = pl < BK && pb + pl < p_end;
            const int h0 = q_h[l] * g.sH - g.pH, w0 = q_w[l] * g.sW - g.pW;
            ra[l] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (VEC) {
                const int h = h0 + ti[0], w = w0 + tj[0];
                if (p_ok && e_ok[0] && (unsigned)h < (unsigned)g.H && (unsigned)w < (unsigned)g.W)
                    ra[l] = __ldg(reinterpret_cast<const float4*>(x0 + (long long)((q_s[l] * g.H + h) * g.W + w) * g.Cin + tc[0]));
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int h = h0 + ti[e], w = w0 + tj[e];
                    if (p_ok && e_ok[e] && (unsigned)h < (unsigned)g.H && (unsigned)w < (unsigned)g.W)
                        reinterpret_cast<float*>(&ra[l])[e] = __ldg(x0 + (long long)((q_s[l] * g.H + h) * g.W + w) * g.Cin + tc[e]);
                }
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
                if (VEC) {
                    if (n < g.Cout) rb[l] = __ldg(reinterpret_cast<const float4*>(p));
                } else {
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (n + q < g.Cout) reinterpret_cast<float*>(&rb[l])[q] = __ldg(p + q);
                }
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
    if (iters > 0) {
        load_tile();
        store_tile(0);
        __syncthreads();
    }
    for (int it = 0; it < iters; ++it) {
        if (it + 1 < iters) load_tile();
        simt_fma_tile<BM, BN, TM, TN>(As[it & 1], Bs[it & 1], ty, tx, acc);
        if (sum_dy) {
#pragma unroll
            for (int k = 0; k < BK; ++k) bsum += Bs[it & 1][k][tid];
        }
        if (it + 1 < iters) {
            store_tile((it + 1) & 1);
            __syncthreads();
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
template <int BM, int BN, int TM, int TN, bool DX>
static int launch_simt_conv(const SimtGemm& g, long long M, int classes, bool vec, cudaStream_t st) {
    const int ntn = ceil_div(g.N, BN);
    const long long mt = (M + BM - 1) / BM;
    if (mt * ntn > 0x7fffffffLL) return set_error(AE_UNSUPPORTED, "convolution of %lld pixels and %d channels is too large", M, g.N);
    const dim3 grid((unsigned)(mt * ntn), 1, (unsigned)classes);
    constexpr int THREADS = (BM / TM) * (BN / TN);
    if (vec) launch(simt_conv_kernel<BM, BN, TM, TN, DX, true>, grid, THREADS, 0, st, g, ntn);
    else launch(simt_conv_kernel<BM, BN, TM, TN, DX, false>, grid, THREADS, 0, st, g, ntn);
    count_launch();
    return check_launch("simt_conv_kernel");
}

// Tile of the forward pass and dX: the one whose busiest SM is through first.  An SM takes as many CTAs at a time as its
// registers hold (`ctas`) and works at `rate` then (relative, measured: 8x8 sums per thread reach up to 63 TFLOP/s over the chip, 4x4 28); with
// fewer it waits for latency, which is why few pixels take the small tiles.
struct SimtTile { int bm, bn, ctas; double rate; };
static constexpr SimtTile SIMT_CONV_TILES[] = {{128, 128, 2, 0.8}, {128, 64, 3, 1.0},  {64, 64, 6, 0.95},
                                               {128, 32, 4, 0.7}, {128, 16, 4, 0.42}, {64, 32, 4, 0.45}};
static int simt_pick_tile(const SimtTile* tiles, int n, long long M, int N, long long copies) {
    int best = 0;
    double best_cost = 1e300;
    for (int i = 0; i < n; ++i) {
        const SimtTile& t = tiles[i];
        const long long count = (M + t.bm - 1) / t.bm * ceil_div(N, t.bn) * copies;
        const long long per_sm = (count + num_sms() - 1) / num_sms(), rest = per_sm % t.ctas;
        double cost = (double)(per_sm - rest);
        if (rest) cost += rest / (0.1 + 0.9 * rest / t.ctas);
        cost *= t.bm * (double)t.bn / t.rate;
        if (cost < best_cost) { best_cost = cost; best = i; }
    }
    return best;
}

template <bool DX>
static int simt_conv(const SimtGemm& g, long long M, int classes, bool vec, cudaStream_t st) {
    switch (simt_pick_tile(SIMT_CONV_TILES, 6, M, g.N, classes)) {
        case 0: return launch_simt_conv<128, 128, 8, 8, DX>(g, M, classes, vec, st);
        case 1: return launch_simt_conv<128, 64, 8, 8, DX>(g, M, classes, vec, st);
        case 2: return launch_simt_conv<64, 64, 8, 8, DX>(g, M, classes, vec, st);
        case 3: return launch_simt_conv<128, 32, 8, 4, DX>(g, M, classes, vec, st);
        case 4: return launch_simt_conv<128, 16, 4, 4, DX>(g, M, classes, vec, st);
        default: return launch_simt_conv<64, 32, 4, 4, DX>(g, M, classes, vec, st);
    }
}

int simt_conv_fwd(const AetherConvDesc& d, const float* x, const float* w, const float* b, float* y, cudaStream_t st) {
    SimtGemm g{};
    int Ho, Wo;
    conv_out_hw(d, Ho, Wo);
    g.in = x; g.w = w; g.bias = b; g.out = y;
    g.IH = d.H; g.IW = d.W; g.IC = d.Cin; g.N = d.Cout;
    g.fH = d.fH; g.fW = d.fW; g.sH = d.sH; g.sW = d.sW; g.pH = d.padH; g.pW = d.padW;
    g.OH = Ho; g.OW = Wo; g.S = d.S; g.Cin = d.Cin; g.Cout = d.Cout;
    const bool vec = d.Cin % 4 == 0 && d.Cout % 4 == 0 && aligned16(x) && aligned16(w) && aligned16(y);
    return simt_conv<false>(g, 1LL * d.S * Ho * Wo, 1, vec, st);
}

int simt_conv_bwd_data(const AetherConvDesc& d, const float* dy, const float* w, float* dx, cudaStream_t st) {
    SimtGemm g{};
    int Ho, Wo;
    conv_out_hw(d, Ho, Wo);
    g.in = dy; g.w = w; g.out = dx;
    g.IH = Ho; g.IW = Wo; g.IC = d.Cout; g.N = d.Cin;
    g.fH = d.fH; g.fW = d.fW; g.sH = d.sH; g.sW = d.sW; g.pH = d.padH; g.pW = d.padW;
    g.OH = d.H; g.OW = d.W; g.S = d.S; g.Cin = d.Cin; g.Cout = d.Cout;
    const bool vec = d.Cin % 4 == 0 && d.Cout % 4 == 0 && aligned16(dy) && aligned16(w) && aligned16(dx);
    const long long M = 1LL * d.S * ceil_div(d.H, d.sH) * ceil_div(d.W, d.sW);     // pixels of the largest class
    if (1LL * d.sH * d.sW > 65535) return set_error(AE_UNSUPPORTED, "stride %dx%d is too large", d.sH, d.sW);
    return simt_conv<true>(g, M, d.sH * d.sW, vec, st);
}

// Tile and split of dW: the tile whose padded filter entries x output channels cost least at the rate of its thread tile, and
// as many splits of the pixels as fill the chip, each at least 16 steps long so that its partial is worth writing.
static constexpr SimtTile SIMT_DW_TILES[] = {{128, 128, 2, 1.0}, {128, 64, 3, 0.97}, {96, 64, 4, 0.9},
                                             {64, 64, 6, 0.85},   {64, 32, 4, 0.6},  {32, 64, 4, 0.6}};
struct SimtDwPlan {
    int tile, tiles_k, tiles_n, splits;
    long long per_split;
};
static SimtDwPlan simt_dw_plan(const AetherConvDesc& d) {
    int Ho, Wo;
    conv_out_hw(d, Ho, Wo);
    SimtDwPlan p;
    const int KK = d.fH * d.fW * d.Cin;
    const long long P = 1LL * d.S * Ho * Wo;
    double best = 1e300;
    for (int i = 0; i < (int)(sizeof(SIMT_DW_TILES) / sizeof(SimtTile)); ++i) {
        const SimtTile& t = SIMT_DW_TILES[i];
        const double cost = 1.0 * ceil_div(KK, t.bm) * t.bm * ceil_div(d.Cout, t.bn) * t.bn / t.rate;
        if (cost < best) { best = cost; p.tile = i; }
    }
    p.tiles_k = ceil_div(KK, SIMT_DW_TILES[p.tile].bm);
    p.tiles_n = ceil_div(d.Cout, SIMT_DW_TILES[p.tile].bn);
    const int per_sm = SIMT_DW_TILES[p.tile].ctas;
    long long want = (long long)per_sm * num_sms() / (1LL * p.tiles_k * p.tiles_n);
    const long long most = (P + 16 * SIMT_BK - 1) / (16 * SIMT_BK);
    if (want > most) want = most;
    if (want < 1) want = 1;
    if (want > 65535) want = 65535;
    p.per_split = ((P + want - 1) / want + SIMT_BK - 1) / SIMT_BK * SIMT_BK;
    p.splits = (int)((P + p.per_split - 1) / p.per_split);
    return p;
}

size_t simt_conv_workspace_bytes(const AetherConvDesc& d) {
    const size_t entries = (size_t)d.fH * d.fW * d.Cin * d.Cout + d.Cout;
    return align_up((size_t)simt_dw_plan(d).splits * entries * sizeof(float), 1024);
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
    if (!ws || ws_bytes < simt_conv_workspace_bytes(d))
        return set_error(AE_BAD_ARG, "conv workspace too small: %zu < %zu", ws_bytes, simt_conv_workspace_bytes(d));
    const SimtDwPlan p = simt_dw_plan(d);
    SimtDw g{};
    conv_out_hw(d, g.Ho, g.Wo);
    g.x = dw ? x : nullptr; g.dy = dy; g.part = static_cast<float*>(ws);
    g.S = d.S; g.H = d.H; g.W = d.W; g.Cin = d.Cin; g.Cout = d.Cout; g.fW = d.fW;
    g.sH = d.sH; g.sW = d.sW; g.pH = d.padH; g.pW = d.padW;
    g.KK = d.fH * d.fW * d.Cin;
    g.P = 1LL * d.S * g.Ho * g.Wo;
    g.per_split = p.per_split;
    const bool vec = d.Cin % 4 == 0 && d.Cout % 4 == 0 && aligned16(x) && aligned16(dy);
    switch (p.tile) {
        case 0: launch_simt_dw<128, 128, 8, 8>(g, p, vec, st); break;
        case 1: launch_simt_dw<128, 64, 8, 8>(g, p, vec, st); break;
        case 2: launch_simt_dw<96, 64, 8, 8>(g, p, vec, st); break;
        case 3: launch_simt_dw<64, 64, 8, 8>(g, p, vec, st); break;
        case 4: launch_simt_dw<64, 32, 4, 4>(g, p, vec, st); break;
        default: launch_simt_dw<32, 64, 4, 4>(g, p, vec, st); break;
    }
    int rc = check_launch("simt_dw_kernel");
    if (rc) return rc;
    return smallc_reduce_partials(g.part, p.splits, g.KK, d.Cout, dw, db, st);
}

}  // namespace aether
