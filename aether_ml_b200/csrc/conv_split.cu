// Single-precision convolution on the tensor cores: every fp32 operand is the sum of three bf16 numbers (8 + 8 + 8 bits of
// mantissa, exponents of the same range), x = x0 + x1 + x2 with x0 = bf16(x), x1 = bf16(x - x0), x2 = bf16(x - x0 - x1), and a
// product of two fp32 numbers the six products x0 w0, x0 w1, x1 w0, x0 w2, x1 w1, x2 w0 (what is left out is below 2^-25 of it).  It
// serves what the kernels on plain bf16 / TF32 operands do not take and the CUDA cores took (conv_simt.cu): AETHER_MATH_FP32,
// strided layers, channel counts that are no multiple of 4 -- forward, dX and dW as implicit GEMMs (CNN_classes_cupy.py:70-154).
//
// Accuracy.  tcgen05 adds in fp32 but truncates after every step of 16 products (measured: one step keeps 25 fractional bits; the
// error of a plain bf16 sum of 2048 exact products is 2.1e-6 and biased, 18 times an FMA loop's), so a sum stays in TMEM for
// four steps only: the x0 w0 products of each stage go to an accumulator of their own that the epilogue warps add to their running
// sums in registers (rounding to nearest) while the next stages are multiplied.  The products of second and third
// order are 2^-8 and 2^-16 of that and stay in two accumulators of their own for up to EPOCH_STAGES stages.  Relative error against
// float64, FMA kernels / this one: 96 x 28x28 32->64 y 3.0e-7 / 7.8e-8, dX 4.2e-7 / 9.5e-8, dW 3.8e-7 / 1.4e-7, and smaller in
// all of forty drawn layers on N(0, 1) and in ten with x positive.  Where every product has one sign truncation always loses: there y 2.3e-7 / 6.8e-8,
// dX 3.2e-7 / 9.1e-8, but dW 6.0e-8 / 8.9e-8, at worst 1.7 times the FMAs' error (dW of 6 x 43x43 88->188 1x1 5.2e-8 / 8.4e-8).  Sums taken out every
// two steps lower that (dW 6.4e-8), but round more often (dW of N(0, 1) 1.6e-7, of 24 x 28x28 128->128 5x5 2.5e-7 -> 3.4e-7) and cost 2-3 %.  An
// output that is not finite (an infinite or NaN operand has no meaningful remainder) is summed again by FMAs from the fp32 arrays.
//
// Time.  Six MMAs take the place of one, 1/6 of the bf16 rate is 3.7 times the FMA pipes'.  N columns of the filter (dy in dW) are
// staged as [w0 | w1 | w2], so that x0 multiplies [w1 | w2] and x1 [w0 | w1] in one MMA of 2 N columns each: four MMAs
// per step, of whose operands shared memory delivers 4 x 4 KB + 6 N x 32 B against 6 N / 2 tensor clocks.  The
// parts are made by a pass over x and dy (split3_kernel: 4 bytes read, 6 written, dB on the way) and copied by TMA, rows of 64
// channels with zeros behind the last: channel counts need not be multiples of anything.  A strided layer's x is stored by
// phases, so that a tap's pixels lie side by side (element strides in the tensor map halve the copies' rate).
// Measured on B200, forward + backward, CUDA cores / this file: 40 x 33x32 64->128 442 / 131 us, 96 x 28x28 32->64 207 / 100, 100 x 57x45
// 48->72 stride 2 431 / 187 (one set of inputs; three in turn, as a program's arrays come: 211 / 104, 433 / 206).  No counter is saturated: the
// tensor pipe is 24-48 % busy, L1 and shared memory 40-67 %, DRAM 6-31 %.  By the clock, the MMAs take 224 for a step of 64 columns by themselves (28 KB of
// operands) and 340 with the copies' writes beside them (18 KB a step): some 150 bytes per clock through shared memory, forward, dX and dW alike, although its
// counters show room.  What holds a step up there is not settled.  Not the number of threads that issue and not the stores (two teams of summing warps and products
// spread over two threads: no change); all sums of a stage side by side in 192 columns: 30 -> 35-39 us, TMEM gives some 110 bytes per clock beside the MMAs.
#include <string.h>

#include <cuda_bf16.h>

#include <type_traits>

#include "common.cuh"
#include "sm100_ptx.cuh"
#include "tc_host.cuh"

namespace aether {

static constexpr int EPOCH_STAGES = 32;         // stages after which the small products' sums leave TMEM, too
static constexpr int SPLIT_EPI_WARPS = 8;       // 4 TMEM lane quarters x 2 (16-column blocks taken in turn)
static constexpr int SPLIT_THREADS = 128 + 32 * SPLIT_EPI_WARPS;     // warps 0 and 1 copy, 2 and 3 multiply, the others add and store
static constexpr int DW_PIXELS = 64;            // pixel rows per stage of dW
// Operands are multiplied by 2^24 before they are split and sums by 2^-48 when they are stored: the lowest bit of the smallest subnormal
// number is then 2^-125, so no part of a fp32 number is subnormal in bf16 (without it operands below 2^-109 lost bits: error 1.6e-7 at
// 2^-112, 2.2e-6 at 2^-116, 3.5e-5 at 2^-120, everything at 2^-140).  Operands from 2^104 on, and sums from 2^80 on, come out infinite and are
// summed again by FMAs.
static constexpr float SPLIT_SCALE = 16777216.f, SPLIT_UNSCALE = 1.f / (SPLIT_SCALE * SPLIT_SCALE);

// Quotients by a number known at launch (Granlund and Montgomery, Division by Invariant Integers using Multiplication, 1994: a multiplication,
// an addition and a shift; dividends below 2^31): the roles of the kernel decode their units by them
// again and again, and an integer division is some 40 instructions.
struct SplitDiv {
    uint32_t d, mul, shift;
};
static SplitDiv split_div(uint32_t d) {
    uint32_t shift = 0;
    while ((1ull << shift) < d) ++shift;
    return {d, (uint32_t)((((1ull << shift) - d) << 32) / d + 1), shift};
}
__device__ __forceinline__ int split_quot(int n, const SplitDiv& d) { return (int)((__umulhi((uint32_t)n, d.mul) + (uint32_t)n) >> d.shift); }

// A pixel class of dX: output rows h = hs + a * sH see the taps i = ph + ti * sH at input row a + hq - ti.  (Forward: one class.)
struct SplitClass {
    int16_t ph, pw, nH, nW, hs, ws, hq, wq;
    int MH, MW;
};
static constexpr int SPLIT_MOST_STRIDE = 4;

struct SplitParams {
    CUtensorMap tm_a;     // igemm: pixels (C, W, H, N, part x phase), box KC x BW x BH x BN; dW: x
    CUtensorMap tm_b;     // igemm: filter (K, columns, part x tap), box KC x NT; dW: dy (C, W, H, N, part)
    const float* in;      // the fp32 arrays behind them, for outputs that are not finite; dW: x
    const float* w;       // filter (taps, Cin, Cout); dW: dy
    const float* bias;    // nullable
    float* out;           // dW: partial sums [split][U][KC][ldn]
    int* status;
    int IH, IW, IC;       // extent of `in`
    int OH, OW, S;        // extent of the output pixels (dW: of dy)
    int N;                // output columns
    int fH, fW, sH, sW, pH, pW, Cin, Cout;
    int dx;               // gather over dy, a stride's input pixels in sH * sW classes
    int BW, BH, BN, rows, tiles_w, tiles_h, tiles_n;
    int NT, n_tiles_n;    // column tile (a multiple of 16; dW: 64 or 128)
    int kchunks, last_ksteps;
    int units;
    SplitDiv by_ntn, by_tiles, by_tw, by_th, by_groups;     // column tiles, pixel tiles, tile columns, tile rows, groups of row units
    SplitClass cls[SPLIT_MOST_STRIDE * SPLIT_MOST_STRIDE];
    int U, cblocks, splits, ksteps, ldn;      // dW: units of KC filter rows (tap, KC channels), pixel splits, steps per stage
};

// KC: channels per row of a tile, 64 or 32 (64-byte swizzle).  A stage is KC channels of a tap or, in dW, a box of pixels: at most four steps
// of 16 products, whose x0 w0 sum leaves TMEM then.
template <int NTMAX, bool DW, int KC>
struct SplitCfg {
    static constexpr int ROW = KC * 2;                                      // bytes
    static constexpr int UNITS = 128 / KC;                                  // dW: row units of the 128 accumulator rows
    static constexpr int A_PART = DW ? UNITS * DW_PIXELS * ROW : 128 * ROW; // one part of the 128 accumulator rows' operand
    static constexpr int STAGE_A = 3 * A_PART;
    static constexpr int STAGE_B = 3 * NTMAX * (DW ? 2 * DW_PIXELS : ROW);  // (dW: tiles of 64 channels of dy)
    static constexpr int FIT = (216 * 1024) / (STAGE_A + STAGE_B), STAGES = FIT < 6 ? FIT : 6;
    static constexpr int SMEM_BYTES = 1024 + STAGES * (STAGE_A + STAGE_B) + 256;
    static constexpr int NBG = NTMAX <= 64 ? 4 : 2;             // accumulators of a stage's x0 w0
    static constexpr int NBC = NTMAX <= 64 ? 2 : 1;             // accumulator pairs of the small products
    static constexpr int BLOCKS = NTMAX / 32;                   // 16-column blocks of an epilogue warp
    static_assert((NBG + NBC * 2) * NTMAX <= 512 && STAGES >= 2, "TMEM, shared memory");
};

// Row (column) offset `a` of a tap against stride `s`: the phase of the input pixels it reads, and where in them.
__device__ __forceinline__ void split_phase(int a, int s, int& phase, int& at) {
    at = a >= 0 ? a / s : -((-a + s - 1) / s);
    phase = a - at * s;
}

// Pixel tile `t` of p's tiling: first column, row and image.
__device__ __forceinline__ void split_tile_origin(const SplitParams& p, int t, int& w0, int& h0, int& n0) {
    const int a = split_quot(t, p.by_tw), n = split_quot(a, p.by_th);
    w0 = (t - a * p.tiles_w) * p.BW;
    h0 = (a - n * p.tiles_h) * p.BH;
    n0 = n * p.BN;
}

// Unit -> column tile; igemm: pixel tile `mt` of class `cls`; dW: group of row units `mt`, range of pixel tiles [t0, t1) of split `cls`.
template <bool DW>
__device__ __forceinline__ void split_unit(const SplitParams& p, int u, int& nt, int& mt, int& cls, int& t0, int& t1) {
    const int a = split_quot(u, p.by_ntn);
    nt = u - a * p.n_tiles_n;
    if (DW) {
        const long long ptiles = p.by_tiles.d;
        cls = split_quot(a, p.by_groups);
        mt = a - cls * (int)p.by_groups.d;
        t0 = (int)(ptiles * cls / p.splits);
        t1 = (int)(ptiles * (cls + 1) / p.splits);
    } else {
        cls = split_quot(a, p.by_tiles);
        mt = a - cls * (int)p.by_tiles.d;
        t0 = t1 = 0;
    }
}

// Row `r` of a unit's 128, pixel (b, a, n) of its box: where it goes (null: nowhere) and what it is (igemm: output column, row, image;
// dW: filter column, filter row, channel).
template <bool DW, int KC>
__device__ __forceinline__ float* split_row(const SplitParams& p, int mt, int cls, const SplitClass& c, int w0, int h0, int n0, int r, int b, int a,
                                            int n, int& x_w, int& x_h, int& x_n) {
    if (DW) {
        const int unit = mt * (128 / KC) + r / KC, tap = unit / p.cblocks;
        x_h = tap / p.fW;
        x_w = tap - x_h * p.fW;
        x_n = (unit - tap * p.cblocks) * KC + r % KC;
        return (unit < p.U && x_n < p.Cin) ? p.out + (((size_t)cls * p.U + unit) * KC + r % KC) * p.ldn : nullptr;
    }
    const int w = w0 + b, h = h0 + a;
    x_n = n0 + n;
    x_h = p.dx ? c.hs + h * p.sH : h;
    x_w = p.dx ? c.ws + w * p.sW : w;
    return (r < p.rows && h < c.MH && w < c.MW && x_n < p.S) ? p.out + (((size_t)x_n * p.OH + x_h) * p.OW + x_w) * p.N : nullptr;
}

// Outputs that are not finite, again by FMAs from the fp32 arrays, in the order of the reduction: a plain tiled product by the whole block, in
// the shared memory of the pipeline, after that has ended -- however long it takes, nobody waits for it with a limit.  Blocks of 64 rows x
// 64 columns that have such an output, steps of 32 channels (dW: a box of pixels), 16 x 16 threads with 4 x 4 sums each.  Sums that are NaN stay so:
// when no other is left the block of outputs is done.  Padding is zeros that are multiplied like other pixels (0 * inf), but in dX, which
// has none.  96 x 28x28 32->64, forward / backward, us: finite values 34 / 71, NaN throughout 229 / 417, infinite ones of one sign 610 / 1812, one
// infinite value 172 / 876 (by the lanes that stored them, one output after the other, dW alone some 20 ms by estimate; by rows of a warp and columns of its
// lanes 222 / 535, 1147 / 3105, 90 / 794).  What it costs other passes is in dW's kernel, 1.4 us of 103 for the layer's forward and backward: with an empty body for dW
// that is gone, with one for the other passes not; registers, the form of the call and the size of the body make no difference.
__device__ __forceinline__ bool split_finite(float v) { return fabsf(v) <= 3.402823466e38f; }

template <bool DW, int KC>
__device__ __forceinline__ void split_repair(const SplitParams& p, int nt, int mt, int cls, int t0, int t1, int row0, int col0, float* smem) {
    constexpr int WARPS = SPLIT_THREADS / 32, STEP = DW ? DW_PIXELS : 32, LD = 68;
    float *A = smem, *B = A + STEP * LD;                     // [step][row], [step][column]
    int* pix = reinterpret_cast<int*>(B + STEP * LD);        // column, row and image of pixel r of a box: pix[r], pix[128 + r], pix[256 + r]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, ty = tid >> 4, tx = tid & 15;
    const int last = min((nt + 1) * p.NT, p.N);              // columns [col0, last)
    const SplitClass& c = p.cls[DW ? 0 : cls];
    int w0 = 0, h0 = 0, n0 = 0;
    if (!DW) split_tile_origin(p, mt, w0, h0, n0);
    __syncthreads();                                         // (the outputs before these have been read)
    if (tid < 128) {
        pix[tid] = tid % p.BW;
        pix[128 + tid] = tid / p.BW % p.BH;
        pix[256 + tid] = tid / (p.BW * p.BH);
    }
    __syncthreads();
    // this thread's outputs: rows row0 + 4 ty + m, columns col0 + 4 tx + e
    auto out_row = [&](int m) {
        const int r = row0 + ty * 4 + m;
        int x_w, x_h, x_n;
        return split_row<DW, KC>(p, mt, cls, c, w0, h0, n0, r, pix[r], pix[128 + r], pix[256 + r], x_w, x_h, x_n);
    };
    uint32_t bad = 0;
    if (tid < 256) {
#pragma unroll 1
        for (int m = 0; m < 4; ++m) {
            const float* row = out_row(m);
#pragma unroll 1
            for (int e = 0; e < 4 && row != nullptr; ++e)
                if (col0 + tx * 4 + e < last && !split_finite(row[col0 + tx * 4 + e])) bad |= 1u << (4 * m + e);
        }
    }
    float acc[4][4] = {};
    bool open = bad != 0;
    auto multiply = [&](uint32_t rows) {                     // `rows`: those that the products belong to
        __syncthreads();
        if (tid >= 256) return;
#pragma unroll 1
        for (int k = 0; k < STEP; ++k) {
            const float4 a4 = *reinterpret_cast<const float4*>(A + k * LD + ty * 4), b4 = *reinterpret_cast<const float4*>(B + k * LD + tx * 4);
            const float a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
            for (int m = 0; m < 4; ++m)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float s = fmaf(a[m], b[e], acc[m][e]);
                    acc[m][e] = !DW && !(rows >> m & 1) ? acc[m][e] : s;
                }
        }
        open = false;
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int e = 0; e < 4; ++e) open |= (bad >> (4 * m + e) & 1) && acc[m][e] == acc[m][e];
    };
    if constexpr (DW) {
        for (int t = t0; t < t1; ++t) {
            if (!__syncthreads_or(open)) break;
            split_tile_origin(p, t, w0, h0, n0);
#pragma unroll 1
            for (int r = warp; r < DW_PIXELS; r += WARPS) {
                const int w = w0 + pix[r], h = h0 + pix[128 + r], n = n0 + pix[256 + r];
                const bool ok = r < p.rows && w < p.OW && h < p.OH && n < p.S;
#pragma unroll
                for (int g = 0; g < 64; g += 32) {
                    const int unit = mt * (128 / KC) + (row0 + g) / KC, tap = unit / p.cblocks, i = tap / p.fW;
                    const int ch = (unit - tap * p.cblocks) * KC + (row0 + g) % KC + lane;
                    const int a = h * p.sH - p.pH + i, b = w * p.sW - p.pW + tap - i * p.fW, col = col0 + g + lane;
                    const bool in = ok && (unsigned)a < (unsigned)p.IH && (unsigned)b < (unsigned)p.IW && ch < p.Cin && unit < p.U;
                    const bool in_d = ok && col < last;
                    const float x = __ldg(p.in + (in ? (((size_t)n * p.IH + a) * p.IW + b) * p.Cin + ch : 0));
                    const float d = __ldg(p.w + (in_d ? (((size_t)n * p.OH + h) * p.OW + w) * p.Cout + col : 0));
                    A[r * LD + g + lane] = in ? x : 0.f;
                    B[r * LD + g + lane] = in_d ? d : 0.f;
                }
            }
            multiply(0xfu);
        }
    } else {
        // input pixel (a, b) that row r of the tile sees at filter row i, column j; whether it is one
        auto seen = [&](int r, int i, int j, int& a, int& b) {
            const int h = h0 + pix[128 + r], w = w0 + pix[r];
            a = p.dx ? h + c.hq - (i - c.ph) / p.sH : h * p.sH - p.pH + i;
            b = p.dx ? w + c.wq - (j - c.pw) / p.sW : w * p.sW - p.pW + j;
            return (unsigned)a < (unsigned)p.IH && (unsigned)b < (unsigned)p.IW && n0 + pix[256 + r] < p.S;
        };
        const int i_step = p.dx ? p.sH : 1, j_step = p.dx ? p.sW : 1;
        bool more = true;
        for (int i = p.dx ? c.ph : 0; i < p.fH && more; i += i_step)
            for (int j = p.dx ? c.pw : 0; j < p.fW && more; j += j_step) {
                const float* f = p.w + (size_t)(i * p.fW + j) * p.Cin * p.Cout;
                uint32_t rows = 0;
#pragma unroll 1
                for (int m = 0; m < 4; ++m) {
                    int a, b;
                    rows |= (uint32_t)(!p.dx || seen((row0 + ty * 4 + m) & 127, i, j, a, b)) << m;
                }
                for (int k0 = 0; k0 < p.IC; k0 += STEP) {
                    more = __syncthreads_or(open);
                    if (!more) break;
                    const int k = k0 + lane;
#pragma unroll 2
                    for (int r = warp; r < 64; r += WARPS) {
                        int a, b;
                        const bool in = seen(row0 + r, i, j, a, b) && k < p.IC;
                        const float v = __ldg(p.in + (in ? (((size_t)(n0 + pix[256 + row0 + r]) * p.IH + a) * p.IW + b) * p.IC + k : 0));
                        A[lane * LD + r] = in ? v : 0.f;
                    }
#pragma unroll 2
                    for (int u = warp; u < 64; u += WARPS) {              // the filter's contiguous index on the lanes
                        const int kk = p.dx ? lane : u >> 1, n = p.dx ? u : (u & 1) * 32 + lane;
                        const bool in = k0 + kk < p.IC && col0 + n < last;
                        const float v = __ldg(f + (in ? p.dx ? (size_t)(col0 + n) * p.Cout + k0 + kk : (size_t)(k0 + kk) * p.Cout + col0 + n : 0));
                        B[kk * LD + n] = in ? v : 0.f;
                    }
                    multiply(rows);
                }
            }
    }
    if (bad == 0) return;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        float* row = out_row(m);
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (bad >> (4 * m + e) & 1) row[col0 + tx * 4 + e] = acc[m][e] + (!DW && p.bias != nullptr ? p.bias[col0 + tx * 4 + e] : 0.f);
    }
}

// ... of all units of this block.
template <bool DW, int KC>
__device__ __noinline__ void split_repair_units(const SplitParams& p, float* smem) {
    for (int u = blockIdx.x; u < p.units; u += gridDim.x) {
        int nt, mt, cls, t0, t1;
        split_unit<DW>(p, u, nt, mt, cls, t0, t1);
        for (int row0 = 0; row0 < 128; row0 += 64)
            for (int col0 = nt * p.NT; col0 < min((nt + 1) * p.NT, p.N); col0 += 64) split_repair<DW, KC>(p, nt, mt, cls, t0, t1, row0, col0, smem);
    }
}

// Persistent over units: igemm, a (pixel class, pixel tile, column tile); dW, a (group of row units, column tile, range of pixel tiles).
template <int NTMAX, bool DW, int KC>
__global__ void __launch_bounds__(SPLIT_THREADS, 1) split_conv_kernel(const __grid_constant__ SplitParams p) {
    using Cfg = SplitCfg<NTMAX, DW, KC>;
    constexpr int STAGES = Cfg::STAGES, NBG = Cfg::NBG, NBC = Cfg::NBC, STAGE = Cfg::STAGE_A + Cfg::STAGE_B;
    constexpr int UNITS = Cfg::UNITS;
    constexpr int TILE = DW_PIXELS * Cfg::ROW, DY_TILE = DW_PIXELS * 128, DY_TILES = NTMAX / 64;      // dW: KC channels of x, 64 channels of dy of a box of pixels
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t sBar = smem_base + STAGES * STAGE;
    auto full_bar = [&](int s) { return sBar + 8u * s; };
    auto empty_bar = [&](int s) { return sBar + 8u * (STAGES + s); };
    auto gfull_bar = [&](int b) { return sBar + 8u * (2 * STAGES + b); };                 // the x0 w0 sum of a stage is complete / taken
    auto gempty_bar = [&](int b) { return sBar + 8u * (2 * STAGES + NBG + b); };
    auto cfull_bar = [&](int b) { return sBar + 8u * (2 * STAGES + 2 * NBG + b); };       // an epoch's small products
    auto cempty_bar = [&](int b) { return sBar + 8u * (2 * STAGES + 2 * NBG + NBC + b); };
    const uint32_t sTmemPtr = sBar + 8u * (2 * STAGES + 2 * NBG + 2 * NBC);
    uint8_t* gen_base = smem_raw + (smem_base - smem_u32(smem_raw));
    volatile uint32_t* tmem_ptr_generic = reinterpret_cast<volatile uint32_t*>(gen_base + (sTmemPtr - smem_base));
    volatile uint32_t* repair_flag = tmem_ptr_generic + 1;         // whether this block stored something that is not finite

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;

    if (DW && p.rows < p.ksteps * 16) {
        // rows of a box past p.rows are never written by TMA but read by the last step: zeros
        auto clear = [&](int first, int tiles, int tile_bytes, int row) {
            const int per_tile = (p.ksteps * 16 - p.rows) * (row / 16);                   // 16-byte pieces
            for (int i = threadIdx.x; i < tiles * per_tile; i += SPLIT_THREADS) {
                const int tile = i / per_tile;
                *reinterpret_cast<uint4*>(gen_base + first + (size_t)tile * tile_bytes + p.rows * row + (i - tile * per_tile) * 16) = make_uint4(0, 0, 0, 0);
            }
        };
        for (int s = 0; s < STAGES; ++s) {
            clear(s * STAGE, Cfg::STAGE_A / TILE, TILE, Cfg::ROW);
            clear(s * STAGE + Cfg::STAGE_A, Cfg::STAGE_B / DY_TILE, DY_TILE, 128);
        }
        fence_proxy_async_smem();
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(full_bar(s), 2); mbar_init(empty_bar(s), 2); }
        for (int b = 0; b < NBG; ++b) { mbar_init(gfull_bar(b), 1); mbar_init(gempty_bar(b), SPLIT_EPI_WARPS); }
        for (int b = 0; b < NBC; ++b) { mbar_init(cfull_bar(b), 1); mbar_init(cempty_bar(b), SPLIT_EPI_WARPS); }
        mbar_fence_init();
        *repair_flag = 0;
        tma_prefetch_desc(&p.tm_a);
        tma_prefetch_desc(&p.tm_b);
    }
    if (warp == 3) {
        tmem_alloc(sTmemPtr, 512);
        tmem_relinquish();
    }
    pdl_wait();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_ptr_generic;
    const uint32_t tmem_c = tmem_base + NBG * NTMAX;           // accumulators of the small products

    const int NT = p.NT;
    const int b_part = DW ? DY_TILES * DY_TILE : NT * Cfg::ROW;                       // bytes of one part of the columns' operand
    auto decode = [&](int u, int& nt, int& mt, int& cls, int& t0, int& t1) { split_unit<DW>(p, u, nt, mt, cls, t0, t1); };
    // stages of a unit, and steps of one of them
    auto unit_stages = [&](int cls, int t0, int t1) {
        if (DW) return t1 - t0;
        const SplitClass& c = p.cls[DW ? 0 : cls];
        return c.nH * c.nW * p.kchunks;
    };
    auto stage_steps = [&](int kc) { return DW ? p.ksteps : kc == p.kchunks - 1 ? p.last_ksteps : KC / 16; };

    if (warp < 2) {
        // ---- copies: warp 0 the rows' operand, warp 1 the columns' (warp-uniform loops, one lane issues: see the products)
        const bool leader = elect_one();
        auto copies = [&](auto rows_tag) {
            constexpr bool ROWS = decltype(rows_tag)::value;
            uint32_t s = 0, ph = 0;
            const uint32_t tx = 3u * (DW ? (uint32_t)p.rows * (ROWS ? 256u : DY_TILES * 128u) : (uint32_t)(ROWS ? p.rows : NT) * Cfg::ROW);
            const int phases = p.dx ? 1 : p.sH * p.sW;
            auto free_stage = [&] { return __all_sync(0xffffffffu, mbar_wait_spin(empty_bar(s), ph ^ 1u, p.status, DS_TIMEOUT_EMPTY)) != 0; };
            for (int u = blockIdx.x; u < p.units; u += gridDim.x) {
                int nt, mt, cls, t0, t1, w0, h0, n0;
                decode(u, nt, mt, cls, t0, t1);
                if (DW) {
                    int uc[UNITS], uw[UNITS], uh[UNITS], uf[UNITS];       // channel, column, row and phase of the group's units
#pragma unroll
                    for (int k = 0; k < UNITS; ++k) {
                        int unit = mt * UNITS + k, fh, fw;
                        if (unit >= p.U) unit = p.U - 1;          // padding unit of the last group: results are dropped
                        const int tap = unit / p.cblocks, i = tap / p.fW;
                        uc[k] = (unit - tap * p.cblocks) * KC;
                        split_phase(tap - i * p.fW - p.pW, p.sW, fw, uw[k]);
                        split_phase(i - p.pH, p.sH, fh, uh[k]);
                        uf[k] = fh * p.sW + fw;
                    }
                    split_tile_origin(p, t0, w0, h0, n0);
                    for (int t = t0; t < t1; ++t) {
                        if (!free_stage()) return;
                        const uint32_t bar = full_bar(s), at = smem_base + s * STAGE + (ROWS ? 0 : Cfg::STAGE_A);
                        if (leader) {
                            mbar_arrive_expect_tx(bar, tx);
#pragma unroll
                            for (int q = 0; q < 3; ++q) {
                                if (ROWS) {
#pragma unroll
                                    for (int k = 0; k < UNITS; ++k)
                                        tma_load_5d(at + q * Cfg::A_PART + k * TILE, &p.tm_a, bar, uc[k], w0 + uw[k], h0 + uh[k], n0, q * phases + uf[k]);
                                } else {
#pragma unroll
                                    for (int k = 0; k < DY_TILES; ++k) tma_load_5d(at + (q * DY_TILES + k) * DY_TILE, &p.tm_b, bar, nt * NT + 64 * k, w0, h0, n0, q);
                                }
                            }
                        }
                        if (++s == STAGES) { s = 0; ph ^= 1u; }
                        w0 += p.BW;                               // the next tile
                        if (w0 >= p.tiles_w * p.BW) { w0 = 0; h0 += p.BH; }
                        if (h0 >= p.tiles_h * p.BH) { h0 = 0; n0 += p.BN; }
                    }
                } else {
                    // taps in order; forward: phase (fh, fw) and offset (ch, cw) of the input pixels advance with them
                    const SplitClass& c = p.cls[DW ? 0 : cls];
                    split_tile_origin(p, mt, w0, h0, n0);
                    const int iters = c.nH * c.nW * p.kchunks, taps = p.fH * p.fW;
                    int fh = 0, fw = 0, ch = h0 + c.hq, cw = w0 + c.wq, fw0, cw0;
                    if (!p.dx) {
                        split_phase(-p.pH, p.sH, fh, ch);
                        split_phase(-p.pW, p.sW, fw, cw);
                        ch += h0;
                        cw += w0;
                    }
                    fw0 = fw;
                    cw0 = cw;
                    int kc = 0, j = 0, row = c.ph * p.fW, tap = row + c.pw;
                    for (int it = 0; it < iters; ++it) {
                        if (!free_stage()) return;
                        const uint32_t bar = full_bar(s), at = smem_base + s * STAGE + (ROWS ? 0 : Cfg::STAGE_A);
                        if (leader) {
                            mbar_arrive_expect_tx(bar, tx);
#pragma unroll
                            for (int q = 0; q < 3; ++q) {
                                if (ROWS) tma_load_5d(at + q * Cfg::A_PART, &p.tm_a, bar, kc * KC, cw, ch, n0, q * phases + fh * p.sW + fw);
                                else tma_load_3d(at + q * b_part, &p.tm_b, bar, kc * KC, nt * NT, q * taps + tap);
                            }
                        }
                        if (++kc == p.kchunks) {
                            kc = 0;
                            if (p.dx) { --cw; tap += p.sW; }
                            else { ++tap; if (++fw == p.sW) { fw = 0; ++cw; } }
                            if (++j == c.nW) {
                                j = 0;
                                fw = fw0;
                                cw = cw0;
                                if (p.dx) { --ch; row += p.sH * p.fW; }
                                else { row += p.fW; if (++fh == p.sH) { fh = 0; ++ch; } }
                                tap = row + c.pw;
                            }
                        }
                        if (++s == STAGES) { s = 0; ph ^= 1u; }
                    }
                }
            }
        };
        if (warp == 0) copies(std::true_type{});
        else copies(std::false_type{});
        __syncwarp();
    } else if (warp < 4) {
        // ---- products: warp 3 has x0 w0, warp 2 the small ones.  Issuing an MMA or a commit costs a thread about 50 clocks and each
        // barrier it waits for 80, as much as 128 columns take to multiply: with two threads those run beside the MMAs.  The loops
        // are warp-uniform (every lane polls, one issues): descriptors stay in uniform registers, where MMAs take them from.
        const bool main = warp == 3, leader = elect_one();
        const uint32_t idesc1 = make_idesc(1u, DW, DW, 128u, (uint32_t)NT), idesc2 = make_idesc(1u, DW, DW, 128u, 2u * (uint32_t)NT);
        // a step of 16 in units of 16 bytes: 32 bytes along the rows; dW: 16 rows
        constexpr uint32_t ADV = DW ? Cfg::ROW : 2, ADVB = DW ? 128 : 2;
        constexpr uint32_t SBO = 8 * Cfg::ROW, SBOB = DW ? 1024 : SBO;
        const uint64_t pa = make_smem_desc(0, DW ? TILE : 16, SBO, KC == 64 ? 2 : 4), pb = make_smem_desc(0, DW ? DY_TILE : 16, SBOB, DW || KC == 64 ? 2 : 4);
        const uint32_t hi = (uint32_t)(pa >> 32), hib = (uint32_t)(pb >> 32), lo0 = (uint32_t)pa + (smem_base >> 4);
        const uint32_t lob0 = (uint32_t)pb + ((smem_base + Cfg::STAGE_A) >> 4);
        constexpr uint32_t A_NEXT = Cfg::A_PART / 16;
        const uint32_t b_next = (uint32_t)b_part / 16;
        auto wait = [&](uint32_t bar, uint32_t parity, int code) { return __all_sync(0xffffffffu, mbar_wait_spin(bar, parity, p.status, code)) != 0; };
        uint32_t s = 0, ph = 0, gb = 0, gph = 0;          // gb: accumulator of the stage (main) or of the epoch
        bool ok = true;
        for (int u = blockIdx.x; u < p.units && ok; u += gridDim.x) {
            int nt, mt, cls, t0, t1;
            decode(u, nt, mt, cls, t0, t1);
            const int iters = unit_stages(cls, t0, t1);
            int kc = 0, left = 0;                             // stages that the epoch still takes; 0: start one
            for (int it = 0; it < iters; ++it) {
                const int steps = stage_steps(kc);
                if (++kc == p.kchunks) kc = 0;
                const uint32_t da = lo0 + s * (STAGE / 16), db = lob0 + s * (STAGE / 16);
                if (main) {
                    if (!wait(gempty_bar(gb), gph ^ 1u, DS_TIMEOUT_TMEM_EMPTY)) { ok = false; break; }
                    if (!wait(full_bar(s), ph, DS_TIMEOUT_FULL)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t dg = tmem_base + gb * NTMAX;
                    if (leader) {
#pragma unroll
                        for (int k = 0; k < KC / 16 || (DW && k < 4); ++k)
                            if (k < steps) umma_2hi(dg, da + ADV * k, hi, db + ADVB * k, hib, idesc1, k > 0);
                        umma_commit(gfull_bar(gb));
                        umma_commit(empty_bar(s));
                    }
                    if (++gb == NBG) { gb = 0; gph ^= 1u; }
                } else {
                    uint32_t acc = 1u;
                    if (left == 0) {
                        if (!wait(cempty_bar(gb), gph ^ 1u, DS_TIMEOUT_TMEM_EMPTY)) { ok = false; break; }
                        left = EPOCH_STAGES;
                        acc = 0u;
                    }
                    if (!wait(full_bar(s), ph, DS_TIMEOUT_FULL)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t dc = tmem_c + gb * (2 * NTMAX);
                    const bool last = --left == 0 || it == iters - 1;
                    if (leader) {
#pragma unroll
                        for (int k = 0; k < KC / 16 || (DW && k < 4); ++k) {
                            if (k < steps) {
                                umma_2hi(dc, da + ADV * k, hi, db + b_next + ADVB * k, hib, idesc2, k > 0 ? 1u : acc);       // x0 [w1 | w2]
                                umma_2hi(dc, da + A_NEXT + ADV * k, hi, db + ADVB * k, hib, idesc2, 1u);                     // x1 [w0 | w1]
                                umma_2hi(dc + NT, da + 2 * A_NEXT + ADV * k, hi, db + ADVB * k, hib, idesc1, 1u);            // x2 w0
                            }
                        }
                        if (last) umma_commit(cfull_bar(gb));
                        umma_commit(empty_bar(s));
                    }
                    if (last) {
                        left = 0;
                        if (++gb == NBC) { gb = 0; gph ^= 1u; }
                    }
                }
                if (++s == STAGES) { s = 0; ph ^= 1u; }
            }
        }
        __syncwarp();
    } else {
        // ---- sums: warp (q, part) has accumulator rows [32q, 32q + 32), a row per lane, and the 16-column blocks part, part + 2, ...
        constexpr int BLOCKS = Cfg::BLOCKS;
        const int q = warp & 3, part = (warp - 4) >> 2;
        const uint32_t lane0 = ((uint32_t)(q * 32) << 16) + part * 16;
        int r_w[4], r_h[4], r_n[4];                               // the four rows in the box of pixels that this lane's quad stores
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = q * 32 + (lane & ~3) + j;
            r_w[j] = r % p.BW;
            r_h[j] = r / p.BW % p.BH;
            r_n[j] = r / (p.BW * p.BH);
        }
        uint32_t gb = 0, gph = 0, cb = 0, cph = 0;
        bool ok = true;
        for (int u = blockIdx.x; u < p.units && ok; u += gridDim.x) {
            int nt, mt, cls, t0, t1;
            decode(u, nt, mt, cls, t0, t1);
            const int iters = unit_stages(cls, t0, t1);
            float acc[BLOCKS][16];
#pragma unroll
            for (int b = 0; b < BLOCKS; ++b)
#pragma unroll
                for (int k = 0; k < 16; ++k) acc[b][k] = 0.f;
            auto add = [&](uint32_t t) {          // acc += accumulator at column t  (blocks past NT: other accumulators' columns, never stored)
                uint32_t v[BLOCKS][16];
#pragma unroll
                for (int b = 0; b < BLOCKS; ++b) tmem_ld_32x16(t + lane0 + 32 * b, v[b]);
                tmem_ld_wait();
#pragma unroll
                for (int b = 0; b < BLOCKS; ++b)
#pragma unroll
                    for (int k = 0; k < 16; ++k) acc[b][k] += __uint_as_float(v[b][k]);
            };
            auto release = [&](uint32_t bar) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar);
            };
            int left = EPOCH_STAGES;
            for (int it = 0; it < iters; ++it) {
                if (!mbar_wait_spin(gfull_bar(gb), gph, p.status, DS_TIMEOUT_TMEM_FULL)) { ok = false; break; }
                tc_fence_after();
                add(tmem_base + gb * NTMAX);
                release(gempty_bar(gb));
                if (++gb == NBG) { gb = 0; gph ^= 1u; }
                if (--left == 0 || it == iters - 1) {
                    left = EPOCH_STAGES;
                    if (!mbar_wait_spin(cfull_bar(cb), cph, p.status, DS_TIMEOUT_TMEM_FULL)) { ok = false; break; }
                    tc_fence_after();
                    add(tmem_c + cb * (2 * NTMAX) + NT);          // third order, then second
                    add(tmem_c + cb * (2 * NTMAX));
                    release(cempty_bar(cb));
                    if (++cb == NBC) { cb = 0; cph ^= 1u; }
                }
            }
            if (!ok) break;
            int w0 = 0, h0 = 0, n0 = 0, x_w, x_h, x_n;
            const SplitClass& c = p.cls[DW ? 0 : cls];
            if (!DW) split_tile_origin(p, mt, w0, h0, n0);
            float* rowp[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) rowp[j] = split_row<DW, KC>(p, mt, cls, c, w0, h0, n0, q * 32 + (lane & ~3) + j, r_w[j], r_h[j], r_n[j], x_w, x_h, x_n);
            bool bad = false;
            const bool b1 = lane & 1, b2 = lane & 2;
#pragma unroll
            for (int b = 0; b < BLOCKS; ++b) {
                if ((2 * b + part) * 16 < NT) {
                    // The quad's 4 rows x 16 columns are exchanged so that lane i holds columns 4i .. 4i + 3 of all four rows and the
                    // quad stores 64 bytes of a row at a time: bit 1 of the lane against bit 1 of the column group, then bit 0.
                    float m[4][4];                                // [row][column of this lane's group]
                    float t[2][2][4];                             // [row bit 1 of group .. ] after the first exchange
#pragma unroll
                    for (int g = 0; g < 2; ++g)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float lo = acc[b][4 * g + e], up = acc[b][8 + 4 * g + e];        // groups g and g + 2 of this lane's row
                            const float got = __shfl_xor_sync(0xffffffffu, b2 ? lo : up, 2);
                            t[0][g][e] = b2 ? got : lo;           // rows (lane & 1) and (lane & 1) + 2 of groups (lane & 2) + g
                            t[1][g][e] = b2 ? up : got;
                        }
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float got = __shfl_xor_sync(0xffffffffu, b1 ? t[h][0][e] : t[h][1][e], 1);
                            m[2 * h][e] = b1 ? got : t[h][0][e];
                            m[2 * h + 1][e] = b1 ? t[h][1][e] : got;
                        }
                    const int col = nt * NT + (2 * b + part) * 16 + (lane & 3) * 4;
                    float bias[4] = {0.f, 0.f, 0.f, 0.f};
                    if (!DW && p.bias != nullptr) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) bias[e] = col + e < p.N ? __ldg(p.bias + col + e) : 0.f;
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (rowp[j] == nullptr) continue;
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            bad |= !split_finite(m[j][e]);
                            m[j][e] = fmaf(m[j][e], SPLIT_UNSCALE, bias[e]);
                        }
                        if ((DW ? p.ldn : p.N) % 4 == 0) {
                            if (col < p.N) *reinterpret_cast<float4*>(rowp[j] + col) = make_float4(m[j][0], m[j][1], m[j][2], m[j][3]);
                        } else {
#pragma unroll
                            for (int e = 0; e < 4; ++e)
                                if (col + e < p.N) rowp[j][col + e] = m[j][e];
                        }
                    }
                }
            }
            if (bad) *repair_flag = 1;
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 3) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
    if (*repair_flag != 0) split_repair_units<DW, KC>(p, reinterpret_cast<float*>(gen_base));
}

// ====================================================================================== operands
__device__ __forceinline__ void split3(float v, __nv_bfloat16& a, __nv_bfloat16& b, __nv_bfloat16& c) {
    v *= SPLIT_SCALE;                                    // exact, or infinite from 2^104 on
    a = __float2bfloat16_rn(v);
    const float r = v - __bfloat162float(a);             // exact
    b = __float2bfloat16_rn(r);
    c = __float2bfloat16_rn(r - __bfloat162float(b));
}

// A strided layer's x by phases: [sH * sW][S][ceil(H / sH)][ceil(W / sW)] pixels (those outside the image are zero), so that the pixels a tap
// sees lie side by side.
struct SplitPhases {
    int H, W, sH, sW, PH, PW;
    long long images;                                    // S * PH * PW
    // source row of row `r`, or -1
    __device__ __forceinline__ long long source(long long r) const {
        const long long f = r / images;
        const unsigned i = (unsigned)(r - f * images), a = i / (unsigned)PW, n = a / (unsigned)PH;
        const int w = (int)(i - a * PW) * sW + (int)f % sW, h = (int)(a - n * PH) * sH + (int)f / sW;
        return w < W && h < H ? ((long long)n * H + h) * W + w : -1;
    }
};

// fp32 [rows][C] -> three bf16 arrays [3][rows][Cp] (channels padded with zeros) and, when asked for, each block's
// column sums of the fp32 input (for dB).  Bound by HBM: 4 bytes read, 6 written.
template <bool COLSUM, bool STRIDED>
__device__ __forceinline__ void split3_rows(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, long long rows, int C, int Cp,
                                            float* __restrict__ colsum_part, long long rows_per_block, const SplitPhases& f, int block, float* red) {
    const int G = Cp / 8;                                // groups of eight channels
    const long long r_begin = block * rows_per_block;
    const long long r_end = r_begin + rows_per_block < rows ? r_begin + rows_per_block : rows;
    const size_t plane = (size_t)rows * Cp;
    for (int gbase = 0; gbase < G; gbase += 256) {
        const int Gc = (G - gbase) < 256 ? (G - gbase) : 256, lanes = 256 / Gc;
        const int g = gbase + threadIdx.x % Gc, rl = threadIdx.x / Gc, c0 = g * 8;
        float acc[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] = 0.f;
        if (rl < lanes) {
            const bool whole = C % 4 == 0 && c0 + 8 <= C;
            constexpr int U = 4;                         // rows in flight
            for (long long r0 = r_begin + rl; r0 < r_end; r0 += U * lanes) {
                float v[U][8];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const long long r = r0 + u * lanes;
                    const long long at = STRIDED && r < r_end ? f.source(r) : r;
                    const float* s = src + at * C + c0;
#pragma unroll
                    for (int k = 0; k < 8; ++k) v[u][k] = 0.f;
                    if (r < r_end && at >= 0) {
                        if (whole) {
                            *reinterpret_cast<float4*>(v[u]) = __ldcs(reinterpret_cast<const float4*>(s));
                            *reinterpret_cast<float4*>(v[u] + 4) = __ldcs(reinterpret_cast<const float4*>(s + 4));
                        } else {
#pragma unroll
                            for (int k = 0; k < 8; ++k)
                                if (c0 + k < C) v[u][k] = __ldg(s + k);
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const long long r = r0 + u * lanes;
                    if (r < r_end) {
                        __align__(16) __nv_bfloat16 o[3][8];
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            if (COLSUM) acc[k] += v[u][k];
                            split3(v[u][k], o[0][k], o[1][k], o[2][k]);
                        }
#pragma unroll
                        for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4*>(dst + q * plane + (size_t)r * Cp + c0) = *reinterpret_cast<const uint4*>(o[q]);
                    }
                }
            }
        }
        if (COLSUM) {
#pragma unroll
            for (int k = 0; k < 8; ++k) red[threadIdx.x * 8 + k] = acc[k];
            __syncthreads();
            for (int cc = threadIdx.x; cc < Gc * 8; cc += 256) {
                const int c = gbase * 8 + cc;
                if (c < C) {
                    float s = 0.f;
                    for (int l = 0; l < lanes; ++l) s += red[(l * Gc + cc / 8) * 8 + cc % 8];
                    colsum_part[(size_t)block * C + c] = s;
                }
            }
            __syncthreads();
        }
    }
}

// The filter's operands from one read of w (taps, Cin, Cout): fwd [3][taps][Cout][Cin_p] (transposed), dx [3][taps][Cin][Cout_p].
// Tile `b` of 32 x 32 channels: output channels fastest, then input channels, then taps.
__device__ __forceinline__ void split3_filter_tile(const float* __restrict__ w, __nv_bfloat16* __restrict__ fwd, __nv_bfloat16* __restrict__ dx,
                                                   int taps, int Cin, int Cout, int Cin_p, int Cout_p, int b, float (*tile)[33]) {
    const int nt = (Cout_p + 31) / 32, kt = (Cin_p + 31) / 32, q = b / nt, tap = q / kt;
    const int n0 = (b - q * nt) * 32, k0 = (q - tap * kt) * 32, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    auto put = [&](__nv_bfloat16* dst, size_t plane, size_t at, float v) {
        __nv_bfloat16 x, y, z;
        split3(v, x, y, z);
        dst[at] = x;
        dst[at + plane] = y;
        dst[at + 2 * plane] = z;
    };
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int k = k0 + ty + 8 * r, n = n0 + tx;
        const float v = (k < Cin && n < Cout) ? w[((size_t)tap * Cin + k) * Cout + n] : 0.f;
        tile[ty + 8 * r][tx] = v;
        if (dx != nullptr && k < Cin && n < Cout_p) put(dx, (size_t)taps * Cin * Cout_p, ((size_t)tap * Cin + k) * Cout_p + n, v);
    }
    if (fwd == nullptr) return;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int n = n0 + ty + 8 * r, k = k0 + tx;
        if (n < Cout && k < Cin_p) put(fwd, (size_t)taps * Cout * Cin_p, ((size_t)tap * Cout + n) * Cin_p + k, tile[tx][ty + 8 * r]);
    }
}

// The parts of an array and, by the first `filter_blocks` CTAs, of the filter (one launch for what a forward pass needs).
template <bool COLSUM, bool STRIDED>
__global__ void __launch_bounds__(256) split3_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, long long rows, int C,
                                                     int Cp, float* __restrict__ colsum_part, long long rows_per_block, const SplitPhases f,
                                                     const float* __restrict__ w, __nv_bfloat16* __restrict__ fwd, __nv_bfloat16* __restrict__ dx,
                                                     int taps, int Cin, int Cout, int Cin_p, int Cout_p, int filter_blocks) {
    pdl_wait();
    __shared__ float red[COLSUM ? 256 * 8 : 32 * 33];
    if ((int)blockIdx.x < filter_blocks) {
        split3_filter_tile(w, fwd, dx, taps, Cin, Cout, Cin_p, Cout_p, (int)blockIdx.x, reinterpret_cast<float (*)[33]>(red));
        return;
    }
    split3_rows<COLSUM, STRIDED>(src, dst, rows, C, Cp, colsum_part, rows_per_block, f, (int)blockIdx.x - filter_blocks, red);
}

// ====================================================================================== host side
struct SplitPlan {
    bool use;
    int Ho, Wo, taps, Cin_p, Cout_p, PH, PW;      // PH, PW: a phase's extent
    PixelTiling til_fwd, til_dx, til_dw;
    int nt_fwd, nt_dx, nt_dw, kc_in, kc_out, splits, cblocks, U, ldn, db_blocks;
    size_t off_wf, off_wd, off_x, off_dy, off_part, off_dbpart, fwd_total, total;      // (what a forward pass needs lies in front)
};

// The box of at most `most` pixels with the least to do: tiles times rows to the next `unit`, and half a unit for each tile (28x28 in boxes
// of 16 pixels has no rows of padding, but a stage of one step takes 650 clocks and one of three 970).
static PixelTiling split_tiling(int S, int H, int W, int most, int unit) {
    PixelTiling best{};
    long long best_cost = -1;
    for (int bw = 1; bw <= W && bw <= most; ++bw)
        for (int bh = 1; bh <= H && bw * bh <= most; ++bh) {
            int bn = bh < H ? 1 : most / (bw * bh);
            if (bn > S) bn = S;
            const PixelTiling t = {bw, bh, bn, bw * bh * bn, ceil_div(W, bw), ceil_div(H, bh), ceil_div(S, bn)};
            const long long cost = t.total() * (2 * ((t.rows + unit - 1) / unit) + 1);
            if (best_cost < 0 || cost < best_cost || (cost == best_cost && bw > best.BW)) {
                best_cost = cost;
                best = t;
            }
        }
    return best;
}

// Column tile: the one whose rounds over the SMs are through first (a unit's time goes with its columns, but for what the
// 128 rows' copies take).
static int split_nt(int N, long long tiles) {
    int best = 16;
    double best_cost = 1e300;
    for (int nt = 16; nt <= 128; nt += 16) {
        const long long units = tiles * ceil_div(N, nt);
        const double cost = (double)((units + num_sms() - 1) / num_sms()) * (48.0 + nt);
        if (cost < best_cost - 1e-9) { best_cost = cost; best = nt; }
    }
    return best;
}

// Channels per row: 32 where the last 64 would be half empty and few are in front of it.
static int split_kc(int C) { return C <= 96 && ceil_div(C, 32) % 2 == 1 ? 32 : 64; }

static SplitPlan compute_split_plan(const AetherConvDesc& d) {
    SplitPlan pl{};
    conv_out_hw(d, pl.Ho, pl.Wo);
    pl.taps = d.fH * d.fW;
    // Rows of the parts: whole tile rows of 64 or 128 bytes, or a tap's copies take up to twice as long (dX of 100 x 57x45 48->72 stride 2
    // 103 -> 62 us with rows of 128 channels instead of 72); a pointwise layer copies each row once and is better off with less to write.
    pl.kc_in = split_kc(d.Cin);
    pl.kc_out = split_kc(d.Cout);
    const int ui = pl.taps > 1 ? pl.kc_in : 8, uo = pl.taps > 1 ? pl.kc_out : 8;
    pl.Cin_p = (d.Cin + ui - 1) / ui * ui;
    pl.Cout_p = (d.Cout + uo - 1) / uo * uo;
    if (d.sH > SPLIT_MOST_STRIDE || d.sW > SPLIT_MOST_STRIDE || pl.taps > 64 || d.padH > 16384 || d.padW > 16384) return pl;
    if (d.Cin < 16 || d.Cout < 16) return pl;
    // Short reductions: nothing to gain in accuracy over the FMA kernels' (their error grows with the reduction, this one's does not).
    if (pl.taps * d.Cin < 64 || pl.taps * d.Cout < 64) return pl;
    pl.PH = ceil_div(d.H, d.sH);
    pl.PW = ceil_div(d.W, d.sW);
    const size_t in_rows = (size_t)d.sH * d.sW * d.S * pl.PH * pl.PW, out_rows = (size_t)d.S * pl.Ho * pl.Wo;
    if ((in_rows * pl.Cin_p + out_rows * pl.Cout_p) * 6 > (2ull << 30)) return pl;      // (the parts are scratch of the caller's)
    // What the FMA kernels take for a layer (33 TFLOP/s) must be worth the passes that make the parts (5 TB/s) and the longer way
    // through the kernels.  Forward and backward on B200, CUDA cores / split, us: 209 x 23x18 36->16 stride 2 60 / 65, 17 x 13x21
    // 32->16 5x5 36 / 42 and 2 x 9x10 65->130 36 / 47 stay; 6 x 16x16 32->165 5x5 88 / 74, 12 x 24x24 16->146 70 / 50, 6 x 43x43
    // 88->188 1x1 53 / 44, 208 x 53x48 16->64 stride 2 255 / 203, 24 x 18x18 48->208 stride 2 98 / 40, 123 x 18x18 36->46 5x5 532 / 152 go.
    const double fma_us = 6.0 * d.S * pl.Ho * pl.Wo * pl.taps * d.Cin * d.Cout / 33e6;
    const double parts_us = (1.0 * in_rows * (4.0 * d.Cin / (d.sH * d.sW) + 6.0 * pl.Cin_p) + 1.0 * out_rows * (4.0 * d.Cout + 6.0 * pl.Cout_p)) / 5e6;
    if (fma_us < 12.0 + 1.6 * parts_us) return pl;
    if (1LL * d.S * d.H * d.W * ceil_div(d.Cin > d.Cout ? d.Cin : d.Cout, 16) > 0x7fffffffLL) return pl;       // units in 32 bits
    pl.use = true;
    pl.til_fwd = split_tiling(d.S, pl.Ho, pl.Wo, 128, 128);
    pl.til_dx = split_tiling(d.S, pl.PH, pl.PW, 128, 128);
    pl.til_dw = split_tiling(d.S, pl.Ho, pl.Wo, DW_PIXELS, 16);
    pl.nt_fwd = split_nt(d.Cout, pl.til_fwd.total());
    pl.nt_dx = split_nt(d.Cin, pl.til_dx.total() * d.sH * d.sW);
    pl.cblocks = ceil_div(d.Cin, pl.kc_in);
    pl.U = pl.taps * pl.cblocks;
    pl.ldn = (d.Cout + 3) / 4 * 4;
    // dW: 64 or 128 channels of dy per unit.  Copies and operand reads together go at some 150 bytes per clock whichever it is: per
    // step and 128 columns 40 KB of operands and 24 KB of copies, 56 and 36 in two units.  A stage takes 0.74 / 1.16 us, and the partial
    // sums of a split are written and read again: 64 x 28x28 128->128 96 -> 78 us, 40 x 33x32 64->128 5x5 106 -> 82, 100 x 57x45 48->72 stride 2
    // 74 -> 68; 200 x 14x14 72->144 90 -> 94, 16 x 7x7 256->256 16.2 -> 17.5 and 12 x 24x24 16->146 18.5 -> 20.3 stay with 64.
    const long long ptiles = pl.til_dw.total();
    double best = 1e300;
    for (int nt = 64; nt <= (d.Cout > 64 ? 128 : 64); nt += 64) {
        const long long cols = 1LL * ceil_div(pl.U, 128 / pl.kc_in) * ceil_div(d.Cout, nt);
        long long splits = num_sms() / cols;
        if (splits > ptiles / 4) splits = ptiles / 4;
        if (splits < 1) splits = 1;
        const double rounds = (double)((cols * splits + num_sms() - 1) / num_sms());
        const double us = rounds * (double)((ptiles + splits - 1) / splits) * (nt == 64 ? 0.74 : 1.16) + 8.0 * splits * pl.U * pl.kc_in * pl.ldn / 5e6;
        if (us < best) { best = us; pl.nt_dw = nt; pl.splits = (int)splits; }
    }
    pl.db_blocks = (int)(out_rows < 4ull * num_sms() * 64 ? (out_rows + 63) / 64 : 4ull * num_sms());
    size_t off = 0;
    auto take = [&](size_t bytes) { size_t o = off; off = align_up(off + bytes, 1024); return o; };
    pl.off_wf = take((size_t)3 * pl.taps * d.Cout * pl.Cin_p * 2);
    pl.off_wd = take((size_t)3 * pl.taps * d.Cin * pl.Cout_p * 2);
    pl.off_x = take(3 * in_rows * pl.Cin_p * 2);
    pl.fwd_total = off;
    pl.off_dy = take(3 * out_rows * pl.Cout_p * 2);
    pl.off_part = take((size_t)pl.splits * pl.U * pl.kc_in * pl.ldn * 4);
    pl.off_dbpart = take((size_t)pl.db_blocks * d.Cout * 4);
    pl.total = off;
    return pl;
}
static const SplitPlan& split_plan(const AetherConvDesc& d) { return cached_plan<SplitPlan, compute_split_plan>(d); }

bool split_conv_eligible(const AetherConvDesc& d) { return split_plan(d).use; }
size_t split_conv_workspace_bytes(const AetherConvDesc& d) { return split_plan(d).total; }
size_t split_conv_fwd_workspace_bytes(const AetherConvDesc& d) { return split_plan(d).fwd_total; }

// (C, W, H, N, part x phase) bf16, box kc channels x the pixels of `t`.
static int split_pixel_map(CUtensorMap* m, const void* base, int Cp, int W, int H, int N, int phases, const PixelTiling& t, int kc) {
    const cuuint64_t row = (cuuint64_t)Cp * 2;
    const cuuint64_t dims[5] = {(cuuint64_t)Cp, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)N, (cuuint64_t)3 * phases};
    const cuuint64_t strides[4] = {row, row * W, row * W * H, row * W * H * N};
    const cuuint32_t box[5] = {(cuuint32_t)kc, (cuuint32_t)t.BW, (cuuint32_t)t.BH, (cuuint32_t)t.BN, 1};
    const cuuint32_t es[5] = {1, 1, 1, 1, 1};
    return make_map(m, base, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, dims, strides, box, es, kc == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B);
}

template <int NTMAX, bool DW, int KC>
static int launch_split(const SplitParams& p, int prof, cudaStream_t st) {
    using Cfg = SplitCfg<NTMAX, DW, KC>;
    static PerDeviceSmem configured;
    if (int rc = ensure_dynamic_smem(split_conv_kernel<NTMAX, DW, KC>, Cfg::SMEM_BYTES, configured, "split_conv")) return rc;
    const int grid = (int)(p.units < num_sms() ? p.units : num_sms());
    prof_begin(prof, st);
    launch(split_conv_kernel<NTMAX, DW, KC>, grid, SPLIT_THREADS, Cfg::SMEM_BYTES, st, p);
    prof_end(prof, st);
    count_launch();
    return check_launch("split_conv_kernel");
}

static SplitClass split_class(const AetherConvDesc& d, int cls) {
    const int ph = cls / d.sW, pw = cls % d.sW;
    SplitClass c;
    c.ph = (int16_t)ph;
    c.pw = (int16_t)pw;
    c.nH = (int16_t)(ph < d.fH ? (d.fH - ph - 1) / d.sH + 1 : 0);
    c.nW = (int16_t)(pw < d.fW ? (d.fW - pw - 1) / d.sW + 1 : 0);
    const int hs = ((ph - d.padH) % d.sH + d.sH) % d.sH, ws = ((pw - d.padW) % d.sW + d.sW) % d.sW;
    c.hs = (int16_t)hs;
    c.ws = (int16_t)ws;
    c.hq = (int16_t)((hs + d.padH - ph) / d.sH);             // exact (hs + padH = ph mod sH), not negative (ph < sH)
    c.wq = (int16_t)((ws + d.padW - pw) / d.sW);
    c.MH = hs < d.H ? (d.H - hs - 1) / d.sH + 1 : 0;
    c.MW = ws < d.W ? (d.W - ws - 1) / d.sW + 1 : 0;
    return c;
}

static void split_geometry(SplitParams& p, const AetherConvDesc& d, const PixelTiling& t) {
    p.S = d.S; p.fH = d.fH; p.fW = d.fW; p.sH = d.sH; p.sW = d.sW; p.pH = d.padH; p.pW = d.padW; p.Cin = d.Cin; p.Cout = d.Cout;
    p.BW = t.BW; p.BH = t.BH; p.BN = t.BN; p.rows = t.rows; p.tiles_w = t.tiles_w; p.tiles_h = t.tiles_h; p.tiles_n = t.tiles_n;
    p.status = device_status_word();
    p.by_tw = split_div(t.tiles_w);
    p.by_th = split_div(t.tiles_h);
    p.by_tiles = split_div((uint32_t)t.total());
    p.by_ntn = split_div(p.n_tiles_n);
}

// Forward (dx false: in = x, copies of it at `cp`) and dX (in = dy).
static int run_split_igemm(const AetherConvDesc& d, const SplitPlan& pl, bool dx, const float* in, const void* cp, const float* w, const void* wcp,
                           const float* bias, float* out, cudaStream_t st) {
    SplitParams p;
    memset(&p, 0, sizeof(p));
    const PixelTiling& t = dx ? pl.til_dx : pl.til_fwd;
    p.NT = dx ? pl.nt_dx : pl.nt_fwd;
    p.n_tiles_n = ceil_div(dx ? d.Cin : d.Cout, p.NT);
    split_geometry(p, d, t);
    p.in = in; p.w = w; p.bias = bias; p.out = out; p.dx = dx;
    p.IH = dx ? pl.Ho : d.H; p.IW = dx ? pl.Wo : d.W; p.IC = dx ? d.Cout : d.Cin;
    p.OH = dx ? d.H : pl.Ho; p.OW = dx ? d.W : pl.Wo; p.N = dx ? d.Cin : d.Cout;
    for (int k = 0; k < (dx ? d.sH * d.sW : 1); ++k) p.cls[k] = dx ? split_class(d, k) : SplitClass{0, 0, (int16_t)d.fH, (int16_t)d.fW, 0, 0, 0, 0, p.OH, p.OW};
    const int kc = dx ? pl.kc_out : pl.kc_in;
    p.kchunks = ceil_div(p.IC, kc);
    p.last_ksteps = ceil_div(p.IC - (p.kchunks - 1) * kc, 16);
    p.units = (int)(t.total() * p.n_tiles_n * (dx ? d.sH * d.sW : 1));
    const int Cp = dx ? pl.Cout_p : pl.Cin_p;
    if (int rc = split_pixel_map(&p.tm_a, cp, Cp, dx ? pl.Wo : pl.PW, dx ? pl.Ho : pl.PH, d.S, dx ? 1 : d.sH * d.sW, t, kc)) return rc;
    const cuuint64_t dims[3] = {(cuuint64_t)Cp, (cuuint64_t)p.N, (cuuint64_t)3 * pl.taps};
    const cuuint64_t strides[2] = {(cuuint64_t)Cp * 2, (cuuint64_t)Cp * 2 * p.N};
    const cuuint32_t box[3] = {(cuuint32_t)kc, (cuuint32_t)p.NT, 1}, es[3] = {1, 1, 1};
    if (int rc = make_map(&p.tm_b, wcp, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dims, strides, box, es, kc == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B)) return rc;
    const int prof = dx ? PK_IGEMM_DX : PK_IGEMM_FWD;
    if (kc == 32) return p.NT <= 64 ? launch_split<64, false, 32>(p, prof, st) : launch_split<128, false, 32>(p, prof, st);
    return p.NT <= 64 ? launch_split<64, false, 64>(p, prof, st) : launch_split<128, false, 64>(p, prof, st);
}

// The parts of src and, when w is given, of the filter's operands (fwd nullable).
static int launch_split3(const AetherConvDesc& d, const SplitPlan& pl, const float* src, void* dst, long long rows, int C, int Cp, const SplitPhases& f,
                         float* colsum, const float* w, void* fwd, void* dx, cudaStream_t st) {
    const int lanes = Cp / 8 >= 256 ? 1 : 256 / (Cp / 8);
    long long nb = colsum ? pl.db_blocks : 8LL * num_sms();
    if (!colsum && nb * lanes > rows) nb = (rows + lanes - 1) / lanes;
    const int filter = w ? ceil_div(pl.Cout_p, 32) * ceil_div(pl.Cin_p, 32) * pl.taps : 0;
    const auto kernel = colsum ? split3_kernel<true, false> : f.sH * f.sW > 1 ? split3_kernel<false, true> : split3_kernel<false, false>;
    prof_begin(PK_SHADOW, st);
    launch(kernel, (int)nb + filter, 256, 0, st, src, static_cast<__nv_bfloat16*>(dst), rows, C, Cp, colsum, (rows + nb - 1) / nb, f, w,
           static_cast<__nv_bfloat16*>(fwd), static_cast<__nv_bfloat16*>(dx), pl.taps, d.Cin, d.Cout, pl.Cin_p, pl.Cout_p, filter);
    prof_end(PK_SHADOW, st);
    count_launch();
    return check_launch("split3_kernel");
}
// The parts of x, by phases.
static int split_x(const AetherConvDesc& d, const SplitPlan& pl, const float* x, void* dst, const float* w, void* fwd, void* dx, cudaStream_t st) {
    const SplitPhases f = {d.H, d.W, d.sH, d.sW, pl.PH, pl.PW, 1LL * d.S * pl.PH * pl.PW};
    return launch_split3(d, pl, x, dst, f.images * d.sH * d.sW, d.Cin, pl.Cin_p, f, nullptr, w, fwd, dx, st);
}

int split_conv_fwd(const AetherConvDesc& d, const float* x, const float* w, const float* b, float* y, void* ws, cudaStream_t st) {
    const SplitPlan& pl = split_plan(d);
    uint8_t* wsb = static_cast<uint8_t*>(ws);
    if (int rc = split_x(d, pl, x, wsb + pl.off_x, w, wsb + pl.off_wf, wsb + pl.off_wd, st)) return rc;
    return run_split_igemm(d, pl, false, x, wsb + pl.off_x, w, wsb + pl.off_wf, b, y, st);
}

int split_conv_bwd(const AetherConvDesc& d, const float* x, const float* dy, const float* w, float* dx, float* dw, float* db, void* ws,
                   int copies_valid, cudaStream_t st) {
    const SplitPlan& pl = split_plan(d);
    uint8_t* wsb = static_cast<uint8_t*>(ws);
    float* dbpart = reinterpret_cast<float*>(wsb + pl.off_dbpart);
    int rc;
    // (dX's filter operand too, where the forward pass has not left it)
    const bool make_w = dx && !(copies_valid & AETHER_CONV_W_COPY_READY);
    if ((rc = launch_split3(d, pl, dy, wsb + pl.off_dy, 1LL * d.S * pl.Ho * pl.Wo, d.Cout, pl.Cout_p, SplitPhases{0, 0, 1, 1, 0, 0, 0},
                            db ? dbpart : nullptr, make_w ? w : nullptr, nullptr, wsb + pl.off_wd, st)))
        return rc;
    if (dx) {
        if ((rc = run_split_igemm(d, pl, true, dy, wsb + pl.off_dy, w, wsb + pl.off_wd, nullptr, dx, st))) return rc;
    }
    if (!dw) return db ? colsum_finish(dbpart, pl.db_blocks, d.Cout, db, st) : AE_OK;
    if (!(copies_valid & AETHER_CONV_X_COPY_READY) && (rc = split_x(d, pl, x, wsb + pl.off_x, nullptr, nullptr, nullptr, st)))
        return rc;
    SplitParams p;
    memset(&p, 0, sizeof(p));
    const PixelTiling& t = pl.til_dw;
    p.NT = pl.nt_dw;
    p.n_tiles_n = ceil_div(d.Cout, p.NT);
    split_geometry(p, d, t);
    p.in = x; p.w = dy; p.out = reinterpret_cast<float*>(wsb + pl.off_part);
    p.IH = d.H; p.IW = d.W; p.IC = d.Cin; p.OH = pl.Ho; p.OW = pl.Wo; p.N = d.Cout;
    p.U = pl.U; p.cblocks = pl.cblocks; p.splits = pl.splits; p.ldn = pl.ldn;
    p.ksteps = ceil_div(t.rows, 16);
    p.kchunks = 1;
    const int groups = ceil_div(p.U, 128 / pl.kc_in);
    p.by_groups = split_div(groups);
    p.units = groups * p.n_tiles_n * p.splits;
    if ((rc = split_pixel_map(&p.tm_a, wsb + pl.off_x, pl.Cin_p, pl.PW, pl.PH, d.S, d.sH * d.sW, t, pl.kc_in))) return rc;
    if ((rc = split_pixel_map(&p.tm_b, wsb + pl.off_dy, pl.Cout_p, pl.Wo, pl.Ho, d.S, 1, t, 64))) return rc;
    if (p.NT == 64) rc = pl.kc_in == 32 ? launch_split<64, true, 32>(p, PK_DW, st) : launch_split<64, true, 64>(p, PK_DW, st);
    else rc = pl.kc_in == 32 ? launch_split<128, true, 32>(p, PK_DW, st) : launch_split<128, true, 64>(p, PK_DW, st);
    if (rc) return rc;
    return dw_reduce(p.out, dw, p.splits, p.U, pl.kc_in, p.ldn, p.cblocks, pl.taps, d.Cin, d.Cout, pl.taps, p.splits, dbpart, pl.db_blocks, db, st);
}

}  // namespace aether
