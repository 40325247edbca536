// Tensor-core convolution for sm_100a: NHWC implicit GEMM with TMA-staged operand tiles,
// tcgen05.mma accumulating in TMEM, fp32 in/out arrays in the layouts of Aether-ML's Conv_Layer
// (activations NHWC, filters (fH,fW,Cin,Cout); CNN/models/CNN_classes_cupy.py:37-161).
//
//   forward  y[p,d]  = sum_{tap,c} x[p+tap, c] * W[tap,c,d] + b[d]      (einsum at :115, bias :116)
//   dX       dx[p,c] = sum_{tap,d} dy[p-tap, d] * W[tap,c,d]            (einsum :138 + scatter :141-146)
//   dW       dW[tap,c,d] = sum_p x[p+tap, c] * dy[p, d]                 (einsum :134),  dB = sum_p dy (:132)
//
// Nothing is materialised: 'same' padding is the zero fill of out-of-range TMA coordinates, each
// filter tap is a coordinate shift of the same tensor map, and dX is a gather (every dx element is
// written once) instead of the reference's 9x-sized contributions tensor and atomic scatter.
//
// Operand precision: bf16 (kind::f16) on bf16 shadow copies made by a cast kernel, or TF32
// (kind::tf32) straight from the caller's fp32 arrays.  Accumulation is fp32 in TMEM.
#include <stdio.h>
#include <string.h>

#include <cuda_bf16.h>

#include "common.cuh"
#include "finish_columns.cuh"
#include "sm100_ptx.cuh"
#include "pool_epilogue.cuh"
#include "stats_epilogue.cuh"
#include "store_block.cuh"
#include "tc_host.cuh"

namespace aether {

// ====================================================================================== tiling
// Columns of the halo kernel's accumulator: the output channels to the next 32 (the per-tap kernel's tiles are powers of two).
static int halo_n(int out_C, int n_padded) {
    const int n = (out_C + 31) / 32 * 32;
    return n < n_padded ? n : n_padded;
}

static PixelTiling choose_tiling(int S, int H, int W) {
    // Exhaustive search over box shapes with <=128 pixels: minimise the number of tiles (i.e. wasted
    // MMA rows), prefer wide boxes on ties (longer contiguous runs per TMA row).
    PixelTiling best{};
    long long best_tiles = -1;
    for (int bw = 1; bw <= W && bw <= 128; ++bw) {
        for (int bh = 1; bh <= H && bw * bh <= 128; ++bh) {
            int bn = 128 / (bw * bh);
            if (bn > S) bn = S;
            if (bn < 1) continue;
            if (bh < H && bn > 1) continue;  // stack images only once a box covers a whole image height
            long long t = 1LL * ceil_div(W, bw) * ceil_div(H, bh) * ceil_div(S, bn);
            if (best_tiles < 0 || t < best_tiles || (t == best_tiles && bw > best.BW)) {
                best_tiles = t;
                best = PixelTiling{bw, bh, bn, bw * bh * bn, ceil_div(W, bw), ceil_div(H, bh), ceil_div(S, bn)};
            }
        }
    }
    return best;
}

// ====================================================================================== tensor maps
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

int make_map(CUtensorMap* m, const void* base, CUtensorMapDataType dt, int rank, const cuuint64_t* dims, const cuuint64_t* strides,
             const cuuint32_t* box, const cuuint32_t* estr, CUtensorMapSwizzle swz) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return set_error(AE_CUDA, "cuTensorMapEncodeTiled entry point not available");
    CUresult r = fn(m, dt, rank, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
        return set_error(AE_CUDA, "cuTensorMapEncodeTiled(rank %d, %llu x %llu.., box %u x %u..) failed: %d", rank,
                         (unsigned long long)dims[0], (unsigned long long)dims[1], box[0], box[1], (int)r);
    return AE_OK;
}
// NHWC tensor seen as 4-D (C, W, H, N), 128-byte swizzle, box (box_c, BW, BH, BN).
int make_map_nhwc(CUtensorMap* m, const void* base, CUtensorMapDataType dt, int elt, int C, int W, int H, int N, int box_c,
                  int BW, int BH, int BN, CUtensorMapSwizzle swz) {
    const cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)N};
    const cuuint64_t strides[3] = {(cuuint64_t)C * elt, (cuuint64_t)C * elt * W, (cuuint64_t)C * elt * W * H};
    const cuuint32_t box[4] = {(cuuint32_t)box_c, (cuuint32_t)BW, (cuuint32_t)BH, (cuuint32_t)BN};
    const cuuint32_t es[4] = {1, 1, 1, 1};
    return make_map(m, base, dt, 4, dims, strides, box, es, swz);
}
// Row-major matrix (inner = K elements contiguous, `rows` rows), box (box_k, box_rows).
int make_map_2d(CUtensorMap* m, const void* base, CUtensorMapDataType dt, int elt, int inner, long long rows, int box_k,
                int box_rows, CUtensorMapSwizzle swz) {
    const cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)inner * elt};
    const cuuint32_t box[2] = {(cuuint32_t)box_k, (cuuint32_t)box_rows};
    const cuuint32_t es[2] = {1, 1};
    return make_map(m, base, dt, 2, dims, strides, box, es, swz);
}

// ====================================================================================== igemm (forward and dX)
// Pixel tile `t` as column, row and image tile.  32-bit divisions where the count allows (always in practice): four 64-bit
// ones cost the one thread that issues copies 0.3 us per tile, as much as a small layer's tile takes to multiply.
__device__ __forceinline__ void split_tile(long long t, long long total, int tiles_w, int tiles_h, int& tw, int& th, int& tn) {
    if (total <= 0x7fffffffLL) {
        const unsigned u = (unsigned)t, a = u / (unsigned)tiles_w;
        tw = (int)(u - a * (unsigned)tiles_w);
        tn = (int)(a / (unsigned)tiles_h);
        th = (int)(a - (unsigned)tn * (unsigned)tiles_h);
    } else {
        const long long a = t / tiles_w;
        tw = (int)(t - a * tiles_w);
        tn = (int)(a / tiles_h);
        th = (int)(a - (long long)tn * tiles_h);
    }
}

struct IgemmParams {
    CUtensorMap tm_in;   // activations (C, W, H, N), box (128 B of channels, BW, BH, BN)
    CUtensorMap tm_w;    // filter matrix, K contiguous: (K, taps * rows_per_tap), box (128 B of K, NT)
    float* out;          // fp32 output, NHWC (out_N, out_H, out_W, n_out), 16-byte aligned, n_out % 4 == 0
    const float* bias;   // nullable, n_out entries
    float* stats;        // STATS only: [2 * gridDim.x / n_tiles_n][3][n_out] (count, mean, M2) partial rows
    int* status;
    int n_out;
    int out_W, out_H, out_N;   // output extent: accumulator rows outside it are by-products
    int BW, BH, BN, rows;
    int tiles_w, tiles_h, tiles_n, n_tiles_n;
    int rows_per_tap;
    int fH, fW, sgn, off_h, off_w;
    int kchunks;
    int last_ksteps;     // MMAs that the last K chunk of a tap needs
    ActEpilogue act;     // ACT only
    PoolEpilogue pool;   // POOLED only
    int splits;          // SPLIT only: CTAs of a cluster
};

static constexpr int TILE_A_BYTES = 128 * 128;  // 128 pixel rows x 128 B
static constexpr int IGEMM_EPI_WARPS = 8;       // 4 TMEM lane quarters x 2 column halves
static constexpr int IGEMM_EPI_UB = 4;          // 16-column TMEM loads in flight per batch
static constexpr int IGEMM_THREADS = 64 + 32 * IGEMM_EPI_WARPS;   // warp 0 TMA producer, warp 1 MMA issuer, then epilogue
static constexpr int IGEMM_TAIL = 1024;         // barriers, TMEM pointer
static constexpr int IGEMM_STATS_BYTES = IGEMM_EPI_WARPS * STATS_WARP_FLOATS * 4;   // per-warp running column sums and pivots
static constexpr int IGEMM_POOL_CHANNELS = 1024;                                    // most output channels of POOLED, whose coefficients lie there
static_assert(2 * IGEMM_POOL_CHANNELS * 4 <= IGEMM_STATS_BYTES, "coefficients");
static constexpr int IGEMM_SPLIT_BYTES = 4096;                                      // beyond those, SPLIT
static_assert(IGEMM_EPI_WARPS * 2048 <= IGEMM_STATS_BYTES + IGEMM_SPLIT_BYTES, "SPLIT: a warp's 32 x 16 sums of every CTA's epilogue warp");

// PAIR: two CTAs of a cluster share one 256-row MMA (cta_group::2).  Each holds its own 128 pixel rows and HALF of the
// filter tile (NT/2 rows), so a stage is smaller and every SM pulls a third less from L2 per FLOP.
// RB: bytes of K per tile row; 64 (64-byte swizzle, four taps per stage) for layers of at most 32 channels, whose 128-byte rows would be
// half zeros on their way from L2 (896 x 16x16 32->64 31.8 -> 26.2 us, 128 of them 9.5 -> 9.1).
template <int NT, bool PAIR = false, int RB = 128>
struct IgemmCfg {
    static constexpr int B_ROWS = PAIR ? NT / 2 : NT;           // filter rows this CTA stages
    static constexpr int TILE_A_BYTES = 128 * RB;               // 128 pixel rows
    static constexpr int TILE_B_BYTES = B_ROWS * RB;
    // 128-byte K chunks per stage: one thread issues for both SMs of a pair (and the MMAs of narrow tiles are short), and
    // with one chunk per stage its per-stage work (barrier wait, four MMAs, two commits) is not hidden behind the MMAs; a pair's stage takes two
    static constexpr int KS = RB == 64 ? 4 : PAIR || NT <= 64 ? 2 : 1;
    static constexpr int STAGE_A_BYTES = KS * TILE_A_BYTES, STAGE_B_BYTES = KS * TILE_B_BYTES;
    static constexpr int STAGES = RB == 64 ? (NT >= 96 ? 3 : 4) : PAIR ? (NT >= 192 ? 3 : 4) : NT == 256 ? 4 : NT == 192 ? 5 : NT == 128 ? 6 : NT == 96 ? 7 : NT == 64 ? 4 : 5;
    static constexpr int TMEM_COLS = NT == 192 ? 512 : NT == 96 ? 256 : 2 * NT;
    static constexpr int SMEM_BYTES = 1024 + STAGES * (STAGE_A_BYTES + STAGE_B_BYTES) + IGEMM_TAIL + IGEMM_STATS_BYTES;
};

// STATS: the epilogue also accumulates per-channel (count, mean, M2) of the output about the bias, one block per
// CTA group and 32-row quarter; the launch must use a grid that is a multiple of n_tiles_n so that every CTA keeps
// one column tile for all its tiles.
//
// PAIR (launched as clusters of two CTAs): the work unit is a pair of consecutive pixel tiles times one column tile;
// CTA rank r of the pair loads pixel tile 2u + r and filter rows [r * NT/2, (r+1) * NT/2) of the column tile into its
// own shared memory, with the byte counts of both CTAs landing on the even CTA's full barrier.  The even CTA issues
// M = 256 MMAs that read both CTAs' stages and write both CTAs' TMEM (rows of its own pixels, all NT columns), and
// signals both CTAs' barriers; the epilogue warps of both CTAs release the accumulator on the even CTA's barrier.
//
// ACT: the epilogue also writes the (leaky) ReLU of the output and, when asked, the bf16 operand copy of that for the layer
// behind (zero in the padded columns): a Dense layer and its activation of a small network are two launches of two
// microseconds otherwise, three with the cast.
//
// POOLED (inference): Batch_Norm by its running statistics, (leaky) ReLU and 2x2 max pooling in the epilogue, which writes the pooled values and
// their bf16 operand copy only.  Boxes are 8 or 16 pixels wide and an even number of rows high, so that the two rows of a window are 8 or 16 accumulator
// rows apart, in one thread, and its columns in neighbouring ones (lane ^ 4).  (896 x 16x16 32->64 30.8 us, 27.6 and 19.6 apart; 8x8 64->128 20.4, 17.9 and 12.)
//
// SPLIT (one tap, 32 columns): the CTAs of a cluster share the K chunks of one tile, and each adds up, in order of rank, and finishes its part of the
// epilogue warps' sums.  A Dense layer of a small batch is a handful of tiles, each of which pulled all of its rows' K through one SM at 65
// bytes a clock.
template <bool TF32, int NT, bool STATS, bool PAIR, bool ACT = false, int RB = 128, bool POOLED = false, bool SPLIT = false>
__global__ void __launch_bounds__(IGEMM_THREADS, 1) igemm_conv_kernel(const __grid_constant__ IgemmParams p) {
    using Cfg = IgemmCfg<NT, PAIR, RB>;
    static_assert(!SPLIT || (NT == 32 && !PAIR && !STATS && !POOLED), "one batch of columns a warp");
    constexpr int STAGES = Cfg::STAGES, TILE_A_BYTES = Cfg::TILE_A_BYTES;
    constexpr int KC = TF32 ? RB / 4 : RB / 2;    // K elements per row
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t sA = smem_base;
    const uint32_t sB = sA + STAGES * Cfg::STAGE_A_BYTES;
    const uint32_t sBar = sB + STAGES * Cfg::STAGE_B_BYTES;
    // barriers: full[STAGES], empty[STAGES], tmem_full[2], tmem_empty[2]; then the TMEM base address
    auto full_bar = [&](int s) { return sBar + 8u * s; };
    auto empty_bar = [&](int s) { return sBar + 8u * (STAGES + s); };
    auto tfull_bar = [&](int b) { return sBar + 8u * (2 * STAGES + b); };
    auto tempty_bar = [&](int b) { return sBar + 8u * (2 * STAGES + 2 + b); };
    const uint32_t sTmemPtr = sBar + 8u * (2 * STAGES + 4);
    uint8_t* gen_base = smem_raw + (smem_base - smem_u32(smem_raw));   // generic pointer to smem_base
    volatile uint32_t* tmem_ptr_generic =
        reinterpret_cast<volatile uint32_t*>(gen_base + (sTmemPtr - smem_base));

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);      // (warp-uniform for the compiler, too)
    const int lane = threadIdx.x & 31;
    const int cta_rank = PAIR || SPLIT ? (int)cluster_cta_rank() : 0;
    const bool issuer = !PAIR || cta_rank == 0;   // the CTA whose warp 1 issues the MMAs
    const uint32_t gather_bar = sBar + 512, sGather = sBar + IGEMM_TAIL;  // SPLIT: the other CTAs' sums are there (where statistics would be)

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(tfull_bar(b), 1);
            mbar_init(tempty_bar(b), (PAIR ? 2 : 1) * IGEMM_EPI_WARPS);
        }
        if (SPLIT) mbar_init(gather_bar, (p.splits - 1) * (IGEMM_EPI_WARPS / p.splits));
        mbar_fence_init();
        tma_prefetch_desc(&p.tm_in);
        tma_prefetch_desc(&p.tm_w);
    }
    if (warp == 1) {
        if (PAIR) {
            tmem_alloc_pair(sTmemPtr, Cfg::TMEM_COLS);
            tmem_relinquish_pair();
        } else {
            tmem_alloc(sTmemPtr, Cfg::TMEM_COLS);
            tmem_relinquish();
        }
    }
    if (SPLIT) cluster_sync_all();    // the other CTAs' barriers exist before anything is sent to them
    pdl_wait();                       // set-up done; from here on global memory is touched
    float* scale_s = reinterpret_cast<float*>(gen_base + (sBar - smem_base) + IGEMM_TAIL);      // POOLED: scale and shift of all channels
    if (POOLED)
        for (int i = threadIdx.x; i < p.n_out; i += IGEMM_THREADS) pool_coefficients(p.pool, i, p.n_out, scale_s[i], scale_s[IGEMM_POOL_CHANNELS + i]);
    tc_fence_before();
    if (PAIR) cluster_sync_all();     // the other CTA's barriers exist before anything is sent to them
    else __syncthreads();

    tc_fence_after();
    const uint32_t tmem_base = *tmem_ptr_generic;

    // Work units: pixel tiles (PAIR: pairs of consecutive pixel tiles) x column tiles, unit u -> column tile u % n_tiles_n.
    const long long m_tiles = 1LL * p.tiles_w * p.tiles_h * p.tiles_n;
    const long long total_tiles = (PAIR ? (m_tiles + 1) / 2 : m_tiles) * p.n_tiles_n;
    const long long t_first = PAIR ? (blockIdx.x >> 1) : SPLIT ? blockIdx.x / p.splits : blockIdx.x;
    const long long t_step = PAIR ? (gridDim.x >> 1) : SPLIT ? gridDim.x / p.splits : gridDim.x;
    // pixel tile of this CTA in unit t; one past the last tile (odd tile count) decodes to an image index outside the
    // tensor: its loads are zero-filled and none of its rows is stored
    auto decode = [&](long long t, int& nt, int& w0, int& h0, int& n0) {
        long long mt = total_tiles <= 0x7fffffffLL ? (long long)((unsigned)t / (unsigned)p.n_tiles_n) : t / p.n_tiles_n;
        nt = (int)(t - mt * p.n_tiles_n);
        if (PAIR) mt = 2 * mt + cta_rank;
        int tw, th, tn;
        split_tile(mt, m_tiles + 1, p.tiles_w, p.tiles_h, tw, th, tn);
        w0 = tw * p.BW; h0 = th * p.BH; n0 = tn * p.BN;
    };
    const int taps = p.fH * p.fW;
    const int kiters = taps * p.kchunks;
    const int k_begin = SPLIT ? cta_rank * kiters / p.splits : 0, k_end = SPLIT ? (cta_rank + 1) * kiters / p.splits : kiters;
    // bytes per stage on the full barrier: this CTA's two boxes, in a pair those of both CTAs
    const uint32_t chunk_tx = ((uint32_t)p.rows + (uint32_t)Cfg::B_ROWS) * (uint32_t)RB * (PAIR ? 2u : 1u);
    constexpr int KS = Cfg::KS;

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        // One elected lane (elect.sync, not `lane == 0`: the compiler then knows that one thread issues, and a chunk's four
        // MMAs and two copies go out in 130-160 ns instead of 290, less than a 128-column chunk takes to multiply); stages,
        // phases and taps are counted on, not divided out.
        if (elect_one()) {
            uint32_t s = 0, ph = 0;
            bool ok = true;
            for (long long t = t_first; t < total_tiles && ok; t += t_step) {
                int nt, w0, h0, n0;
                decode(t, nt, w0, h0, n0);
                int kc = k_begin, j = 0;                   // the (K chunk, filter column) of the next chunk to load
                int cw = w0 + p.off_w, ch = h0 + p.off_h, wrow = nt * NT + (PAIR ? cta_rank * Cfg::B_ROWS : 0);
                for (int k0 = k_begin; k0 < k_end; k0 += KS) {
                    const int nsub = k_end - k0 < KS ? k_end - k0 : KS;
                    if (!mbar_wait(empty_bar(s), ph ^ 1u, p.status, DS_TIMEOUT_EMPTY)) { ok = false; break; }
                    if (issuer) mbar_arrive_expect_tx(full_bar(s), chunk_tx * (uint32_t)nsub);
                    const uint32_t bar = PAIR ? cluster_map_shared(full_bar(s), 0) : full_bar(s);   // PAIR: the even CTA's
#pragma unroll
                    for (int c = 0; c < KS; ++c) {
                        if (c < nsub) {
                            const uint32_t dA = sA + s * Cfg::STAGE_A_BYTES + c * TILE_A_BYTES;
                            const uint32_t dB = sB + s * Cfg::STAGE_B_BYTES + c * Cfg::TILE_B_BYTES;
                            if (PAIR) {
                                tma_load_4d_pair(dA, &p.tm_in, bar, kc * KC, cw, ch, n0);
                                tma_load_2d_pair(dB, &p.tm_w, bar, kc * KC, wrow);
                            } else {
                                tma_load_4d(dA, &p.tm_in, bar, kc * KC, cw, ch, n0);
                                tma_load_2d(dB, &p.tm_w, bar, kc * KC, wrow);
                            }
                            if (++kc == p.kchunks) {
                                kc = 0;
                                wrow += p.rows_per_tap;
                                cw += p.sgn;
                                if (++j == p.fW) { j = 0; cw = w0 + p.off_w; ch += p.sgn; }
                            }
                        }
                    }
                    if (++s == STAGES) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer (one elected thread)
        if (issuer && elect_one()) {
            constexpr uint32_t idesc = make_idesc(TF32 ? 2u : 1u, 0u, 0u, PAIR ? 256u : 128u, (uint32_t)NT);
            uint32_t s = 0, ph = 0;
            uint32_t lt = 0;
            bool ok = true;
            for (long long t = t_first; t < total_tiles && ok; t += t_step, ++lt) {
                const uint32_t buf = lt & 1u;
                const uint32_t aph = (lt >> 1) & 1u;
                if (!mbar_wait(tempty_bar(buf), aph ^ 1u, p.status, DS_TIMEOUT_TMEM_EMPTY)) { ok = false; break; }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + buf * NT;
                int kc = k_begin;
                for (int k0 = k_begin; k0 < k_end; k0 += KS) {
                    const int nsub = k_end - k0 < KS ? k_end - k0 : KS;
                    if (!mbar_wait(full_bar(s), ph, p.status, DS_TIMEOUT_FULL)) { ok = false; break; }
                    tc_fence_after();
#pragma unroll
                    for (int c = 0; c < KS; ++c) {
                        if (c < nsub) {
                            const uint64_t da = make_smem_desc(sA + s * Cfg::STAGE_A_BYTES + c * TILE_A_BYTES, 16, 8 * RB, RB == 128 ? 2 : 4);
                            const uint64_t db = make_smem_desc(sB + s * Cfg::STAGE_B_BYTES + c * Cfg::TILE_B_BYTES, 16, 8 * RB, RB == 128 ? 2 : 4);
                            const int nk = ++kc == p.kchunks ? p.last_ksteps : RB / 32;
                            if (kc == p.kchunks) kc = 0;
#pragma unroll
                            for (int k = 0; k < RB / 32; ++k) {            // 32 bytes of K each: two 16-byte units further
                                const uint32_t acc = (k0 + c > k_begin || k > 0) ? 1u : 0u;
                                if (k >= nk) break;
                                if (PAIR) umma_pair<TF32>(d_tmem, da + 2u * k, db + 2u * k, idesc, acc);
                                else umma<TF32>(d_tmem, da + 2u * k, db + 2u * k, idesc, acc);
                            }
                        }
                    }
                    // the stage is free (in both CTAs) once these MMAs have read it
                    if (PAIR) {
                        umma_commit_pair(empty_bar(s));
                        umma_commit_pair(cluster_map_shared(empty_bar(s), 1));
                    } else {
                        umma_commit(empty_bar(s));
                    }
                    if (++s == STAGES) { s = 0; ph ^= 1u; }
                }
                if (ok) {
                    if (PAIR) {
                        umma_commit_pair(tfull_bar(buf));
                        umma_commit_pair(cluster_map_shared(tfull_bar(buf), 1));
                    } else {
                        umma_commit(tfull_bar(buf));
                    }
                }
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue (8 warps)
        // Warp (q, part): TMEM lanes [32q, 32q+32), columns [part*NT/2, (part+1)*NT/2).  Accumulators are read with
        // the 16-lane x 256-bit shape and a butterfly exchange inside each quad leaves every lane with 4 consecutive
        // columns of a row, so the registers go straight to global memory as 64-byte pieces per row.
        const int ew = warp - 2;
        const int q = warp & 3;
        const int part = ew >> 2;
        constexpr int ncols = NT / 2;              // columns this warp owns (multiple of 16)
        const int col_begin = part * ncols;
        const int trow = lane >> 2, tcol4 = (lane & 3) * 4;
        const bool lo2 = (lane & 2) == 0, odd = (lane & 1) != 0;
        // statistics: running per-column sums of this warp over all its tiles (stats_epilogue.cuh), memory of its own
        float* stat_w = reinterpret_cast<float*>(gen_base + (sBar - smem_base) + IGEMM_TAIL) + ew * STATS_WARP_FLOATS;
        float st_rows = 0.f;                       // rows (pixels) summed so far, identical in every lane
        if (STATS) {
            for (int i = lane; i < STATS_WARP_FLOATS; i += 32) stat_w[i] = 0.f;
            __syncwarp();
        }
        // The four accumulator rows this thread holds are fixed pixels of the (BW, BH, BN) box.
        int r_w[4], r_h[4], r_n[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = q * 32 + (j >> 1) * 16 + trow + (j & 1) * 8;
            r_w[j] = r % p.BW;
            r_h[j] = (r / p.BW) % p.BH;
            r_n[j] = r < p.rows ? r / (p.BW * p.BH) : (1 << 29);      // rows past the box: never valid
        }
        uint32_t lt = 0;
        bool ok = true;
        for (long long t = t_first; t < total_tiles && ok; t += t_step, ++lt) {
            int nt, w0, h0, n0;
            decode(t, nt, w0, h0, n0);
            const int col0 = nt * NT + col_begin + tcol4;             // first of this thread's columns
            float* rowp[4];
            size_t pix[ACT ? 4 : 1];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int w = w0 + r_w[j], h = h0 + r_h[j], n = n0 + r_n[j];
                const size_t at = ((size_t)n * p.out_H + h) * p.out_W + w;
                rowp[j] = (w < p.out_W && h < p.out_H && n < p.out_N) ? p.out + at * p.n_out + col0 : nullptr;
                if (ACT) pix[ACT ? j : 0] = at;
            }
            long long window = -1;                 // POOLED: the window that this lane finishes
            if (POOLED) {
                const int j = (trow & 1) == 0 ? 0 : p.BW == 16 ? 1 : 2;
                if (rowp[j] != nullptr) window = ((long long)(n0 + r_n[j]) * (p.out_H >> 1) + ((h0 + r_h[j]) >> 1)) * (p.out_W >> 1) + ((w0 + r_w[j]) >> 1);
            }
            float tile_rows = 0.f;                 // valid rows of this tile in this warp's quarter
            if (STATS) {
#pragma unroll
                for (int j = 0; j < 4; ++j) tile_rows += (rowp[j] != nullptr) ? 1.f : 0.f;
                tile_rows += __shfl_xor_sync(0xffffffffu, tile_rows, 4);
                tile_rows += __shfl_xor_sync(0xffffffffu, tile_rows, 8);
                tile_rows += __shfl_xor_sync(0xffffffffu, tile_rows, 16);
            }
            const bool first_stats = STATS && st_rows == 0.f && tile_rows > 0.f;      // the tile that sets the pivots
            const uint32_t buf = lt & 1u;
            const uint32_t aph = (lt >> 1) & 1u;
            if (!mbar_wait(tfull_bar(buf), aph, p.status, DS_TIMEOUT_TMEM_FULL)) { ok = false; break; }
            tc_fence_after();
            const uint32_t taddr0 = tmem_base + ((uint32_t)(q * 32) << 16) + buf * NT + col_begin;
#pragma unroll 1
            for (int cb = 0; cb < ncols; cb += 16 * IGEMM_EPI_UB) {   // batches of IGEMM_EPI_UB x 16 columns
                uint32_t v[2][IGEMM_EPI_UB][8];
                float4 st_s[IGEMM_EPI_UB], st_q[IGEMM_EPI_UB];        // per-column sum / sum of squares of this tile's rows
#pragma unroll
                for (int u = 0; u < IGEMM_EPI_UB; ++u) st_s[u] = st_q[u] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int u = 0; u < IGEMM_EPI_UB; ++u) {
                    if (cb + u * 16 < ncols) {
                        tmem_ld_16x256b_x2(taddr0 + cb + u * 16, v[0][u]);
                        tmem_ld_16x256b_x2(taddr0 + (16u << 16) + cb + u * 16, v[1][u]);
                    }
                }
                tmem_ld_wait();
                if constexpr (SPLIT) {
                    // every CTA adds up and finishes the warps of its rank (mod splits): their registers go to it, [rank][warp][16 bytes of a thread][lane]
                    const int own = ew % p.splits, per = IGEMM_EPI_WARPS / p.splits;
                    const uint32_t slot = (uint32_t)((cta_rank * per + ew / p.splits) * 2048 + lane * 16);
                    if (own != cta_rank) {
                        const uint32_t dst = cluster_map_shared(sGather, own) + slot;
#pragma unroll
                        for (int h = 0; h < 4; ++h) {
                            const uint32_t* q4 = &v[h >> 1][0][(h & 1) * 4];
                            asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + h * 512u), "r"(q4[0]), "r"(q4[1]), "r"(q4[2]), "r"(q4[3]) : "memory");
                        }
                        asm volatile("fence.acq_rel.cluster;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) mbar_arrive_cluster(cluster_map_shared(gather_bar, own));
                        break;
                    }
                    if (!mbar_wait(gather_bar, 0, p.status, DS_TIMEOUT_FULL)) { ok = false; break; }
                    asm volatile("fence.acq_rel.cluster;" ::: "memory");
                    float sum[16];
#pragma unroll
                    for (int e = 0; e < 16; ++e) sum[e] = 0.f;
                    for (int r = 0; r < p.splits; ++r)                // (in order of rank, whichever CTA adds)
#pragma unroll
                        for (int h = 0; h < 4; ++h) {
                            const uint32_t* q4 = &v[h >> 1][0][(h & 1) * 4];
                            float4 o = make_float4(__uint_as_float(q4[0]), __uint_as_float(q4[1]), __uint_as_float(q4[2]), __uint_as_float(q4[3]));
                            if (r != cta_rank)
                                o = *reinterpret_cast<const float4*>(gen_base + (sGather - smem_base) + (r * per + ew / p.splits) * 2048 + h * 512 + lane * 16);
                            sum[4 * h] += o.x; sum[4 * h + 1] += o.y; sum[4 * h + 2] += o.z; sum[4 * h + 3] += o.w;
                        }
#pragma unroll
                    for (int e = 0; e < 16; ++e) v[e >> 3][0][e & 7] = __float_as_uint(sum[e]);
                }
                if (cb + 16 * IGEMM_EPI_UB >= ncols) {           // accumulator fully read by this warp
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if (PAIR) mbar_arrive_cluster(cluster_map_shared(tempty_bar(buf), 0));
                        else mbar_arrive(tempty_bar(buf));
                    }
                }
#pragma unroll
                for (int u = 0; u < IGEMM_EPI_UB; ++u) {
                    if (cb + u * 16 < ncols) {
                        const int cc = cb + u * 16;              // column relative to this thread's first column
                        const bool cols_ok = col0 + cc < p.n_out;   // n_out % 4 == 0: all four columns or none
                        float4 b4 = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (p.bias != nullptr && cols_ok) {
                            b4.x = __ldg(p.bias + col0 + cc + 0); b4.y = __ldg(p.bias + col0 + cc + 1);
                            b4.z = __ldg(p.bias + col0 + cc + 2); b4.w = __ldg(p.bias + col0 + cc + 3);
                        }
                        float4 pv = make_float4(0.f, 0.f, 0.f, 0.f);      // pivot of this lane's four columns
                        if (STATS) pv = *reinterpret_cast<const float4*>(stat_w + 256 + cc + tcol4);
                        float4 act4[POOLED ? 4 : 1], s4 = pv, t4 = pv;
                        if (POOLED && cols_ok) {
                            s4 = *reinterpret_cast<const float4*>(scale_s + col0 + cc);
                            t4 = *reinterpret_cast<const float4*>(scale_s + IGEMM_POOL_CHANNELS + col0 + cc);
                        }
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const uint32_t a0 = v[j >> 1][u][(j & 1) * 2 + 0], a1 = v[j >> 1][u][(j & 1) * 2 + 1];
                            const uint32_t b0 = v[j >> 1][u][4 + (j & 1) * 2 + 0], b1 = v[j >> 1][u][4 + (j & 1) * 2 + 1];
                            // step 1 (lane ^ 2): lanes 0,1 collect column group 0, lanes 2,3 collect group 1
                            const uint32_t s0 = lo2 ? b0 : a0, s1 = lo2 ? b1 : a1;
                            const uint32_t x2 = __shfl_xor_sync(0xffffffffu, s0, 2), x3 = __shfl_xor_sync(0xffffffffu, s1, 2);
                            const uint32_t e0 = lo2 ? a0 : x2, e1 = lo2 ? a1 : x3;       // piece from the even source lane
                            const uint32_t f0 = lo2 ? x2 : b0, f1 = lo2 ? x3 : b1;       // piece from the source lane + 2
                            // step 2 (lane ^ 1): even lanes keep the lower pair of pieces, odd lanes the upper pair
                            const uint32_t t0 = odd ? e0 : f0, t1 = odd ? e1 : f1;
                            const uint32_t g0 = __shfl_xor_sync(0xffffffffu, t0, 1), g1 = __shfl_xor_sync(0xffffffffu, t1, 1);
                            float4 a;                                                     // accumulator values (before the bias)
                            a.x = __uint_as_float(odd ? g0 : e0);
                            a.y = __uint_as_float(odd ? g1 : e1);
                            a.z = __uint_as_float(odd ? f0 : g0);
                            a.w = __uint_as_float(odd ? f1 : g1);
                            if (POOLED) {
                                act4[POOLED ? j : 0] = pool_activation(make_float4(a.x + b4.x, a.y + b4.y, a.z + b4.z, a.w + b4.w), s4, t4, p.pool.alpha);
                                continue;
                            }
                            const bool wr = cols_ok && rowp[j] != nullptr;
                            if (ACT && rowp[j] != nullptr) {
                                const int col = col0 + cc;
                                float4 z = make_float4(a.x + b4.x, a.y + b4.y, a.z + b4.z, a.w + b4.w);
                                z = make_float4(z.x > 0.f ? z.x : p.act.alpha * z.x, z.y > 0.f ? z.y : p.act.alpha * z.y,
                                                z.z > 0.f ? z.z : p.act.alpha * z.z, z.w > 0.f ? z.w : p.act.alpha * z.w);
                                if (!cols_ok) z = make_float4(0.f, 0.f, 0.f, 0.f);
                                else *reinterpret_cast<float4*>(p.act.out + pix[ACT ? j : 0] * p.n_out + col) = z;
                                if (p.act.copy != nullptr && col < p.act.ld) {
                                    const __nv_bfloat162 o[2] = {__floats2bfloat162_rn(z.x, z.y), __floats2bfloat162_rn(z.z, z.w)};
                                    *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.act.copy) + pix[ACT ? j : 0] * p.act.ld + col) =
                                        *reinterpret_cast<const uint2*>(o);
                                }
                            }
                            if (wr)
                                __stcs(reinterpret_cast<float4*>(rowp[j] + cc),
                                       make_float4(a.x + b4.x, a.y + b4.y, a.z + b4.z, a.w + b4.w));
                            if (STATS) {                                     // selects, not products: a by-product may be NaN
                                a.x = wr ? a.x - pv.x : 0.f; a.y = wr ? a.y - pv.y : 0.f;
                                a.z = wr ? a.z - pv.z : 0.f; a.w = wr ? a.w - pv.w : 0.f;
                                st_s[u].x += a.x; st_s[u].y += a.y; st_s[u].z += a.z; st_s[u].w += a.w;
                                st_q[u].x = fmaf(a.x, a.x, st_q[u].x); st_q[u].y = fmaf(a.y, a.y, st_q[u].y);
                                st_q[u].z = fmaf(a.z, a.z, st_q[u].z); st_q[u].w = fmaf(a.w, a.w, st_q[u].w);
                            }
                        }
                        if constexpr (POOLED) {
                            // two windows of two rows here, their other column in lane ^ 4: a lane of an even column finishes the first, of an odd one the second
                            const bool wide = p.BW == 16, right = (trow & 1) != 0;
                            const float4 a_top = act4[0], a_low = wide ? act4[2] : act4[1], b_top = wide ? act4[1] : act4[2], b_low = act4[3];
                            const float4 top = right ? b_top : a_top, low = right ? b_low : a_low, s_top = right ? a_top : b_top, s_low = right ? a_low : b_low;
                            auto other = [](float4 v) {
                                return make_float4(__shfl_xor_sync(0xffffffffu, v.x, 4), __shfl_xor_sync(0xffffffffu, v.y, 4), __shfl_xor_sync(0xffffffffu, v.z, 4),
                                                   __shfl_xor_sync(0xffffffffu, v.w, 4));
                            };
                            const float4 o_top = other(s_top), o_low = other(s_low);
                            const float4 best = right ? pool_first_max(o_top, top, o_low, low) : pool_first_max(top, o_top, low, o_low);
                            if (window >= 0) pool_store(p.pool, window, col0 + cc, p.n_out, best);
                        }
                    }
                }
                if (STATS) {
                    // Lanes with equal lane%4 hold the same 4 columns of 8 different row groups: add them up
                    // (xor 4, 8, 16); lanes 0..3 then add the tile's sums to this warp's running sums in shared
                    // memory (about the column's pivot, see stats_epilogue.cuh).
#pragma unroll
                    for (int m = 4; m <= 16; m <<= 1) {
#pragma unroll
                        for (int u = 0; u < IGEMM_EPI_UB; ++u) {
                            st_s[u].x += __shfl_xor_sync(0xffffffffu, st_s[u].x, m); st_s[u].y += __shfl_xor_sync(0xffffffffu, st_s[u].y, m);
                            st_s[u].z += __shfl_xor_sync(0xffffffffu, st_s[u].z, m); st_s[u].w += __shfl_xor_sync(0xffffffffu, st_s[u].w, m);
                            st_q[u].x += __shfl_xor_sync(0xffffffffu, st_q[u].x, m); st_q[u].y += __shfl_xor_sync(0xffffffffu, st_q[u].y, m);
                            st_q[u].z += __shfl_xor_sync(0xffffffffu, st_q[u].z, m); st_q[u].w += __shfl_xor_sync(0xffffffffu, st_q[u].w, m);
                        }
                    }
                    if (lane < 4) {
#pragma unroll
                        for (int u = 0; u < IGEMM_EPI_UB; ++u) {
                            const int cc = cb + u * 16;
                            if (cc < ncols) stats_fold(stat_w, cc + tcol4, st_s[u], st_q[u], first_stats, tile_rows);
                        }
                    }
                    if (first_stats) __syncwarp();     // the pivots must be visible to the whole warp before its next tile
                }
            }
            st_rows += tile_rows;
        }
        if (STATS) {
            // Two rows (stats_epilogue.cuh) per CTA group: the grid is a multiple of n_tiles_n, so the CTA kept column tile
            // blockIdx.x % n_tiles_n, and the n_tiles_n CTAs of a group fill the disjoint column ranges of rows 2 * group
            // and 2 * group + 1 of [3][n_out].  (PAIR: the same with pairs in the place of CTAs and two rows per CTA of the pair.)
            const int ntc = (int)(t_first % p.n_tiles_n);
            const size_t group = PAIR ? (size_t)(t_first / p.n_tiles_n) * 2 + cta_rank : (size_t)(t_first / p.n_tiles_n);
            stats_merge_store(reinterpret_cast<float*>(gen_base + (sBar - smem_base) + IGEMM_TAIL), ew, lane, st_rows, ncols, ntc * NT, p.n_out,
                              p.bias, p.stats + group * 6 * (size_t)p.n_out);
        }
    }

    tc_fence_before();
    if (PAIR || SPLIT) cluster_sync_all();     // no CTA leaves while another may still address its barriers, memory or TMEM
    else __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        if (PAIR) tmem_dealloc_pair(tmem_base, Cfg::TMEM_COLS);
        else tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
    }
}

// ====================================================================================== dW (filter gradient)
struct DwParams {
    CUtensorMap tm_x;    // (Cin_p, W, H, N), box (128 B of channels, BW, BH, BN)
    CUtensorMap tm_dy;   // (Cout_p, Wo, Ho, N), same box
    float* part;         // [splits][U][UC][ldn] partial sums
    int* status;
    int BW, BH, BN, rows;
    int tiles_w, tiles_h, tiles_n;
    int fH, fW, padH, padW;
    int cblocks;         // 128-byte channel blocks of x
    int U;               // fH*fW*cblocks units (one unit = one tap x one channel block)
    int MG;              // M groups = ceil(U / MB)
    int gpc;             // M groups per CTA
    int n_tiles_n;
    int ldn;
    int Cin, Cout;       // real channels: rows and columns of padding are not stored
};

static constexpr int DW_THREADS = 192;

template <bool TF32, int NB>
struct DwCfg {
    static constexpr int UC = TF32 ? 32 : 64;       // channels per 128-byte block
    static constexpr int MB = 128 / UC;             // x blocks per M=128
    static constexpr int NT = NB * UC;              // dy channels per CTA
    static constexpr int STAGE_BYTES = MB * TILE_A_BYTES;       // x of one M group
    static constexpr int DY_BYTES = NB * TILE_A_BYTES;          // dy of one pixel tile
    static constexpr int DY_STAGES = TF32 ? 2 : NB == 1 ? 4 : 3;        // (a CTA with one M group takes one per stage of x)
    static constexpr int STAGES = (200 * 1024 - DY_STAGES * DY_BYTES) / STAGE_BYTES;
    static constexpr int KROWS = TF32 ? 8 : 16;     // pixel rows per MMA
    static constexpr int SMEM_BYTES = 1024 + STAGES * STAGE_BYTES + DY_STAGES * DY_BYTES + 256;
    static constexpr int MAX_GPC = 512 / NT;
    static_assert(STAGES >= 2, "need at least two stages");
};

// The kernel is bound by what an SM can pull from L2 (some 100 GB/s of it), so a pixel tile's dy is brought in once, in
// stages of its own, and stays for all M groups of the CTA (tf32 256 x 16x16 128->128: 47.5 us with x and dy in one stage per
// group, 44.6 so).
//
// PAIR (clusters of two CTAs, cta_group::2): an M group is 256 rows -- each CTA stages the MB units of its own half --
// and a column tile 2 * NT channels of dy, of which each CTA stages its own NT.  Per stage a CTA loads the same bytes as
// a single CTA but the pair does four times one CTA's products with them: the kernel is bound by what an SM can pull
// from L2, and that halves per FLOP.  p.MG, p.gpc and p.n_tiles_n then count pair groups and pair column tiles.
template <bool TF32, int NB, bool PAIR>
__global__ void __launch_bounds__(DW_THREADS, 1) dw_conv_kernel(const __grid_constant__ DwParams p) {
    using Cfg = DwCfg<TF32, NB>;
    constexpr int STAGES = Cfg::STAGES, MB = Cfg::MB, NT = Cfg::NT, UC = Cfg::UC;
    constexpr int PF = PAIR ? 2 : 1;              // CTAs per M group and column tile
    constexpr int NTP = PF * NT;                  // accumulator columns of one M group
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gen_base = smem_raw + (smem_base - smem_u32(smem_raw));
    constexpr int D = Cfg::DY_STAGES;
    const uint32_t sDy = smem_base + STAGES * Cfg::STAGE_BYTES;
    const uint32_t sBar = sDy + D * Cfg::DY_BYTES;
    auto full_bar = [&](int s) { return sBar + 8u * s; };
    auto empty_bar = [&](int s) { return sBar + 8u * (STAGES + s); };
    auto dfull_bar = [&](int s) { return sBar + 8u * (2 * STAGES + s); };
    auto dempty_bar = [&](int s) { return sBar + 8u * (2 * STAGES + D + s); };
    const uint32_t done_bar = sBar + 8u * (2 * STAGES + 2 * D);
    const uint32_t sTmemPtr = sBar + 8u * (2 * STAGES + 2 * D + 1);
    volatile uint32_t* tmem_ptr_generic = reinterpret_cast<volatile uint32_t*>(gen_base + (sTmemPtr - smem_base));

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);      // (warp-uniform for the compiler, too)
    const int lane = threadIdx.x & 31;
    const int cta_rank = PAIR ? (int)cluster_cta_rank() : 0;
    const bool issuer = cta_rank == 0;

    // Rows of a box past p.rows are never written by TMA; those that belong to the last reduction step are read by the MMAs
    // and must be zero.  Nothing to do when the box is whole steps (clearing all stages took 2 us of a small layer's 11).
    {
        const int k_end = (p.rows + Cfg::KROWS - 1) / Cfg::KROWS * Cfg::KROWS;
        const int per_tile = (k_end - p.rows) * 8;                              // 16-byte pieces
        for (int i = threadIdx.x; i < (STAGES * MB + D * NB) * per_tile; i += blockDim.x) {
            const int tile = i / per_tile;
            *reinterpret_cast<uint4*>(gen_base + (size_t)tile * TILE_A_BYTES + p.rows * 128 + (i - tile * per_tile) * 16) = make_uint4(0, 0, 0, 0);
        }
        fence_proxy_async_smem();
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int s = 0; s < D; ++s) {
            mbar_init(dfull_bar(s), 1);
            mbar_init(dempty_bar(s), 1);
        }
        mbar_init(done_bar, 1);
        mbar_fence_init();
        tma_prefetch_desc(&p.tm_x);
        tma_prefetch_desc(&p.tm_dy);
    }
    if (warp == 1) {
        if (PAIR) {
            tmem_alloc_pair(sTmemPtr, 512);
            tmem_relinquish_pair();
        } else {
            tmem_alloc(sTmemPtr, 512);
            tmem_relinquish();
        }
    }
    pdl_wait();                       // set-up done; from here on global memory is touched
    tc_fence_before();
    if (PAIR) cluster_sync_all();
    else __syncthreads();

    tc_fence_after();
    const uint32_t tmem_base = *tmem_ptr_generic;

    const int split = PAIR ? (blockIdx.x >> 1) : blockIdx.x, splits = PAIR ? (gridDim.x >> 1) : gridDim.x;
    const int gc = blockIdx.y / p.n_tiles_n;
    const int nt = blockIdx.y % p.n_tiles_n;
    const int g_begin = gc * p.gpc;
    const int g_end = min(p.MG, g_begin + p.gpc);
    const int ngroups = g_end - g_begin;
    const long long total_ptiles = 1LL * p.tiles_w * p.tiles_h * p.tiles_n;
    const uint32_t box_tx = (uint32_t)p.rows * 128u * (uint32_t)PF;                           // both CTAs' boxes
    const int ksteps = (p.rows + Cfg::KROWS - 1) / Cfg::KROWS;

    if (warp == 0) {
        if (elect_one()) {                            // (see igemm_conv_kernel)
            struct Unit { int u, cb, i, j; };
            auto unit = [&](int u) { const int tap = u / p.cblocks; return Unit{u, u - tap * p.cblocks, tap / p.fW, tap % p.fW}; };
            auto advance = [&](Unit& x, int n) {
                x.u += n;
                x.cb += n;
                while (x.cb >= p.cblocks) {
                    x.cb -= p.cblocks;
                    if (++x.j == p.fW) { x.j = 0; ++x.i; }
                }
            };
            const Unit first = unit((g_begin * PF + cta_rank) * MB), last = unit(p.U - 1);
            uint32_t s = 0, ph = 0, ds = 0, dph = 0;
            bool ok = true;
            for (long long pt = split; pt < total_ptiles && ok; pt += splits) {
                int tw, th, tn;
                split_tile(pt, total_ptiles, p.tiles_w, p.tiles_h, tw, th, tn);
                const int w0 = tw * p.BW, h0 = th * p.BH, n0 = tn * p.BN;
                if (!mbar_wait(dempty_bar(ds), dph ^ 1u, p.status, DS_TIMEOUT_EMPTY)) break;
                if (issuer) mbar_arrive_expect_tx(dfull_bar(ds), box_tx * (uint32_t)NB);
                const uint32_t dbar = PAIR ? cluster_map_shared(dfull_bar(ds), 0) : dfull_bar(ds);          // PAIR: the even CTA's
#pragma unroll
                for (int nb = 0; nb < NB; ++nb) {
                    const int dyc = ((nt * PF + cta_rank) * NB + nb) * UC;
                    if (PAIR) tma_load_4d_pair(sDy + ds * Cfg::DY_BYTES + nb * TILE_A_BYTES, &p.tm_dy, dbar, dyc, w0, h0, n0);
                    else tma_load_4d(sDy + ds * Cfg::DY_BYTES + nb * TILE_A_BYTES, &p.tm_dy, dbar, dyc, w0, h0, n0);
                }
                if (++ds == D) { ds = 0; dph ^= 1u; }
                Unit x = first;
                for (int g = g_begin; g < g_end; ++g) {
                    if (!mbar_wait(empty_bar(s), ph ^ 1u, p.status, DS_TIMEOUT_EMPTY)) { ok = false; break; }
                    if (issuer) mbar_arrive_expect_tx(full_bar(s), box_tx * (uint32_t)MB);
                    const uint32_t bar = PAIR ? cluster_map_shared(full_bar(s), 0) : full_bar(s);
                    const uint32_t st = smem_base + s * Cfg::STAGE_BYTES;
#pragma unroll
                    for (int m = 0; m < MB; ++m) {
                        const Unit y = x.u < p.U ? x : last;       // padding unit of the last group: results are dropped
                        const int cw = w0 + y.j - p.padW, chh = h0 + y.i - p.padH;
                        if (PAIR) tma_load_4d_pair(st + m * TILE_A_BYTES, &p.tm_x, bar, y.cb * UC, cw, chh, n0);
                        else tma_load_4d(st + m * TILE_A_BYTES, &p.tm_x, bar, y.cb * UC, cw, chh, n0);
                        advance(x, 1);
                    }
                    if (PAIR) advance(x, MB);                      // the other CTA's units
                    if (++s == STAGES) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        if (issuer && elect_one()) {
            constexpr uint32_t idesc = make_idesc(TF32 ? 2u : 1u, 1u, 1u, 128u * PF, (uint32_t)NTP);
            // MN-major operands: 16-bit types use the plain 128-byte swizzle (8-row K groups); 32-bit types need the
            // 32-byte-unit variant (4-row K groups).
            constexpr uint32_t LT = TF32 ? 1u : 2u;
            constexpr uint32_t SBO = TF32 ? 512u : 1024u;
            uint32_t s = 0, ph = 0, ds = 0, dph = 0;
            bool ok = true;
            uint32_t acc0 = 0;
            for (long long pt = split; pt < total_ptiles && ok; pt += splits) {
                if (!mbar_wait(dfull_bar(ds), dph, p.status, DS_TIMEOUT_FULL)) break;
                const uint64_t db0 = make_smem_desc(sDy + ds * Cfg::DY_BYTES, TILE_A_BYTES, SBO, LT);
                for (int g = 0; g < ngroups; ++g) {
                    if (!mbar_wait(full_bar(s), ph, p.status, DS_TIMEOUT_FULL)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t a0 = smem_base + s * Cfg::STAGE_BYTES;
                    uint64_t da = make_smem_desc(a0, TILE_A_BYTES, SBO, LT);
                    uint64_t db = db0;
                    const uint32_t d_tmem = tmem_base + g * NTP;
                    uint32_t acc = acc0;
#pragma unroll 4
                    for (int kk = 0; kk < ksteps; ++kk) {
                        if (PAIR) umma_pair<TF32>(d_tmem, da, db, idesc, acc);
                        else umma<TF32>(d_tmem, da, db, idesc, acc);
                        acc = 1u;
                        da += Cfg::KROWS * 128 / 16;
                        db += Cfg::KROWS * 128 / 16;
                    }
                    if (PAIR) {
                        umma_commit_pair(empty_bar(s));
                        umma_commit_pair(cluster_map_shared(empty_bar(s), 1));
                    } else {
                        umma_commit(empty_bar(s));
                    }
                    if (++s == STAGES) { s = 0; ph ^= 1u; }
                }
                if (ok) {                                          // this tile's dy is free once all groups have used it
                    if (PAIR) {
                        umma_commit_pair(dempty_bar(ds));
                        umma_commit_pair(cluster_map_shared(dempty_bar(ds), 1));
                    } else {
                        umma_commit(dempty_bar(ds));
                    }
                }
                if (++ds == D) { ds = 0; dph ^= 1u; }
                acc0 = 1u;
            }
            if (PAIR) {
                umma_commit_pair(done_bar);
                umma_commit_pair(cluster_map_shared(done_bar, 1));
            } else {
                umma_commit(done_bar);
            }
        }
    } else {
        const int q = warp & 3;
        const bool any_tiles = split < total_ptiles;
        bool ok = true;
        if (any_tiles) ok = mbar_wait(done_bar, 0, p.status, DS_TIMEOUT_TMEM_FULL);
        tc_fence_after();
        if (ok) {
            // this warp's 32 rows belong to one unit: rows c_in0 .. c_in0 + 31 of its channel block
            const int m = q * 32 / UC, c_in0 = q * 32 % UC;
            float* stage = reinterpret_cast<float*>(gen_base) + q * STORE_BLOCK_FLOATS;       // every MMA has read its operands
            for (int g = 0; g < ngroups; ++g) {
                const int u = ((g_begin + g) * PF + cta_rank) * MB + m;
                const int rows = u < p.U ? p.Cin - (u % p.cblocks) * UC - c_in0 : 0;
                float* dst = p.part + (((size_t)split * p.U + u) * UC + c_in0) * (size_t)p.ldn + nt * NTP;
#pragma unroll 1
                for (int ch = 0; ch < NTP / 32; ++ch) {
                    uint32_t r[32];
                    if (any_tiles) {
                        tmem_ld_32x32(tmem_base + ((uint32_t)(q * 32) << 16) + g * NTP + ch * 32, r);
                        tmem_ld_wait();
                    } else {
#pragma unroll
                        for (int k = 0; k < 32; ++k) r[k] = 0u;
                    }
                    store_block_32x32(stage, r, dst + ch * 32, p.ldn, rows, p.Cout - nt * NTP - ch * 32, lane);
                }
            }
        }
    }

    tc_fence_before();
    if (PAIR) cluster_sync_all();
    else __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        if (PAIR) tmem_dealloc_pair(tmem_base, 512);
        else tmem_dealloc(tmem_base, 512);
    }
}

// dW[tap][c][d] = sum over splits of part[split][tap*cblocks + c/UC][c%UC][d]
// Taps from tap_split on have splits2 partials instead of splits (kernels whose CTA classes differ in number).
// V consecutive output channels per thread; 1 << lane_bits threads share an output, thread l of them adds splits l,
// l + lanes, ... and they are combined in fixed order through shared memory (bit-reproducible).  Bound by L2: what counts is
// loads in flight, so lanes are used only where there are few outputs (dw_reduce_lane_bits).
// `nred` CTAs do that; the CTAs behind them finish dB, which saves a launch of its own.
template <int V>
__global__ void __launch_bounds__(256) dw_reduce_kernel(const float* __restrict__ part, float* __restrict__ dw, int splits,
                                                        int U, int UC, int ldn, int cblocks, int taps, int Cin, int Cout,
                                                        int tap_split, int splits2, int lane_bits, int nred,
                                                        const float* __restrict__ dbpart, int db_rows, float* __restrict__ db) {
    pdl_wait();
    __shared__ float4 red4[256];
    if ((int)blockIdx.x >= nred) {                     // the blocks behind: dB from the column sums that came with dy's copy
        finish_columns(dbpart, db_rows, Cout, db, (int)blockIdx.x - nred, reinterpret_cast<float (*)[8]>(red4));
        return;
    }
    const int per = 256 >> lane_bits, lanes = 1 << lane_bits;       // outputs of a CTA, threads per output
    const int el = threadIdx.x & (per - 1), ln = threadIdx.x >> (8 - lane_bits);
    const int Cq = Cout / V;                           // (V == 4: Cout % 4 == 0; ldn a multiple of 4)
    const long long total4 = 1LL * taps * Cin * Cq;
    const size_t split_stride = (size_t)U * UC * ldn;
    for (long long base = 1LL * blockIdx.x * per; base < total4; base += 1LL * nred * per) {
        const long long i4 = base + el;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i4 < total4) {
            const int d = (int)(i4 % Cq) * V;
            const long long tc = i4 / Cq;
            const int c = (int)(tc % Cin);
            const int tap = (int)(tc / Cin);
            const int u = tap * cblocks + c / UC;
            const float* src = part + ((size_t)u * UC + (c % UC)) * (size_t)ldn + d;
            const int ns = tap < tap_split ? splits : splits2;
#pragma unroll 8
            for (int s = ln; s < ns; s += lanes) {
                if constexpr (V == 4) {
                    const float4 v = *reinterpret_cast<const float4*>(src + s * split_stride);
                    acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
                } else {
                    acc.x += src[s * split_stride];
                }
            }
        }
        if (lanes > 1) {
            red4[threadIdx.x] = acc;
            __syncthreads();
            if (ln == 0)
                for (int l = 1; l < lanes; ++l) { const float4 v = red4[l * per + el]; acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w; }
            __syncthreads();
        }
        if (ln == 0 && i4 < total4) {
            if constexpr (V == 4) *reinterpret_cast<float4*>(dw + i4 * 4) = acc;
            else dw[i4] = acc.x;
        }
    }
}

// Threads per output: enough for some 64K threads (128 blocks of 16 warps), at most eight and no more than splits.
static int dw_reduce_lane_bits(long long outputs, int splits) {
    int bits = 0;
    while (bits < 3 && (outputs << bits) < 65536 && (2 << bits) <= splits) ++bits;
    return bits;
}
int dw_reduce(const float* part, float* dw, int splits, int U, int UC, int ldn, int cblocks, int taps, int Cin, int Cout, int tap_split,
              int splits2, const float* dbpart, int db_rows, float* db, cudaStream_t st) {
    const bool v4 = Cout % 4 == 0;
    const long long outputs = 1LL * taps * Cin * (v4 ? Cout / 4 : Cout);
    const int bits = dw_reduce_lane_bits(outputs, splits);
    const long long per = 256 >> bits, groups = (outputs + per - 1) / per, cap = 8LL * num_sms();
    const int nred = (int)(groups < cap ? groups : cap);
    launch(v4 ? dw_reduce_kernel<4> : dw_reduce_kernel<1>, nred + (db ? ceil_div(Cout, 8) : 0), 256, 0, st, part, dw, splits, U, UC, ldn, cblocks,
           taps, Cin, Cout, tap_split, splits2, bits, nred, dbpart, db_rows, db);
    count_launch();
    return check_launch("dw_reduce_kernel");
}

// ====================================================================================== shadow copies
// fp32 [rows][C] -> bf16 [rows][Cp] (zero padded channels).  Optionally also per-block column sums of the
// fp32 input (for dB), written to colsum_part[block][C].
template <bool COLSUM>
__global__ void __launch_bounds__(256) cast_bf16_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst,
                                                        long long rows, int C, int Cp, float* __restrict__ colsum_part,
                                                        long long rows_per_block) {
    pdl_wait();
    const int G = Cp / 8;                 // 8-channel groups per row
    const long long r_begin = blockIdx.x * rows_per_block;
    long long r_end = r_begin + rows_per_block;
    if (r_end > rows) r_end = rows;
    const bool vec = (C % 4) == 0;
    __shared__ float red[COLSUM ? 256 * 8 : 8];
    for (int gbase = 0; gbase < G; gbase += 256) {
        const int Gc = (G - gbase) < 256 ? (G - gbase) : 256;   // groups handled in this pass
        const int planes = 256 / Gc;                            // rows processed concurrently
        const int g = gbase + threadIdx.x % Gc;
        const int plane = threadIdx.x / Gc;
        float acc[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] = 0.f;
        if (plane < planes) {
            const int c0 = g * 8;
            // streaming (evict-first) reads: the fp32 source is not needed again soon, the bf16 copy written here is, so it
            // should be what stays in L2
            const bool whole = vec && c0 + 8 <= C;
            auto take = [&](long long r, const float (&v)[8]) {
                if (COLSUM) {
#pragma unroll
                    for (int k = 0; k < 8; ++k) acc[k] += v[k];
                }
                __nv_bfloat162 o[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) o[k] = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
                *reinterpret_cast<uint4*>(dst + r * Cp + c0) = *reinterpret_cast<uint4*>(o);
            };
            long long r = r_begin + plane;
            if (whole) {
                constexpr int U = 4;                     // rows in flight: eight 16-byte loads per thread
                for (; r < r_end; r += U * planes) {
                    float4 t[U][2];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        if (r + u * planes < r_end) {
                            const float4* s = reinterpret_cast<const float4*>(src + (r + u * planes) * C + c0);
                            t[u][0] = __ldcs(s);
                            t[u][1] = __ldcs(s + 1);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        if (r + u * planes < r_end) {
                            const float v[8] = {t[u][0].x, t[u][0].y, t[u][0].z, t[u][0].w, t[u][1].x, t[u][1].y, t[u][1].z, t[u][1].w};
                            take(r + u * planes, v);
                        }
                    }
                }
            }
            for (; r < r_end; r += planes) {             // (channels of padding, rows that are no multiple of 16 bytes)
                float v[8];
                const float* s = src + r * C + c0;
#pragma unroll
                for (int k = 0; k < 8; ++k) v[k] = (c0 + k < C) ? s[k] : 0.f;
                take(r, v);
            }
        }
        if (COLSUM) {
#pragma unroll
            for (int k = 0; k < 8; ++k) red[threadIdx.x * 8 + k] = acc[k];   // idle threads hold zeros
            __syncthreads();
            for (int cc = threadIdx.x; cc < Gc * 8; cc += blockDim.x) {
                const int c = gbase * 8 + cc;
                if (c < C) {
                    const int gg = cc / 8, k = cc % 8;
                    float s = 0.f;
                    for (int pl = 0; pl < planes; ++pl) s += red[(pl * Gc + gg) * 8 + k];
                    colsum_part[(size_t)blockIdx.x * C + c] = s;
                }
            }
            __syncthreads();
        }
    }
}

// Column sums of an fp32 [rows][C] matrix into part[block][C] (used for dB when no cast pass runs; C % 4 == 0, 16-byte
// aligned).  Four channels per thread, eight rows in flight.
__global__ void __launch_bounds__(256) colsum_kernel(const float* __restrict__ src, long long rows, int C,
                                                     float* __restrict__ part, long long rows_per_block) {
    pdl_wait();
    const long long r_begin = blockIdx.x * rows_per_block;
    long long r_end = r_begin + rows_per_block;
    if (r_end > rows) r_end = rows;
    const int C4 = C >> 2;
    const int cols = C4 < 256 ? C4 : 256;
    const int lanes = 256 / cols;
    __shared__ float4 red[256];
    for (int cbase = 0; cbase < C4; cbase += cols) {
        const int c = cbase + threadIdx.x % cols;
        const int rl = threadIdx.x / cols;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        if (rl < lanes && c < C4) {
            const float4* s = reinterpret_cast<const float4*>(src) + c;
            constexpr int U = 8;                         // (a rest taken one by one would be a round trip each)
            for (long long r = r_begin + rl; r < r_end; r += U * lanes) {
                float4 v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) v[u] = r + u * lanes < r_end ? s[(r + u * lanes) * C4] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int u = 0; u < U; ++u) { acc.x += v[u].x; acc.y += v[u].y; acc.z += v[u].z; acc.w += v[u].w; }
            }
        }
        red[threadIdx.x] = acc;
        __syncthreads();
        if (threadIdx.x < cols && c < C4) {
            for (int l = 1; l < lanes; ++l) { const float4 v = red[l * cols + threadIdx.x]; acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w; }
            reinterpret_cast<float4*>(part + (size_t)blockIdx.x * C)[c] = acc;
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(256) colsum_finish_kernel(const float* __restrict__ part, int nblocks, int C,
                                                            float* __restrict__ out) {
    pdl_wait();
    __shared__ float red[32][8];
    finish_columns(part, nblocks, C, out, (int)blockIdx.x, red);
}

int colsum_finish(const float* part, int rows, int C, float* out, cudaStream_t st) {
    launch(colsum_finish_kernel, ceil_div(C, 8), 256, 0, st, part, rows, C, out);
    count_launch();
    return check_launch("colsum_finish_kernel");
}

// Filter shadows.  w is (taps, Cin, Cout) fp32; the operand copies are zero padded to Cin_p / Cout_p channels.
// They are made through 32 x 32 tiles in shared memory, so that both the reads (consecutive n of w's innermost Cout axis)
// and the writes (consecutive k of the operand's innermost axis) are coalesced; a Dense layer's 8192 x 1024 weight
// matrix goes through here every step.  Writes, from one read of w:
//   fwd (nullable): [tap][Np_f = Cout_p][Kp_f = Cin_p]  = w transposed (forward B operand)
//   dx  (nullable): [tap][Np_d = Cin_p][Kp_d = Cout_p]  = w as it is, padded (dX B operand)
// grid (ceil(Cout_p/32), ceil(Cin_p/32), taps), block (32, 8).
template <typename OutT>
__global__ void __launch_bounds__(256) filter_shadow_tiled_kernel(const float* __restrict__ w, OutT* __restrict__ fwd,
                                                                  OutT* __restrict__ dx, int Cin, int Cout, int Cin_p,
                                                                  int Cout_p) {
    pdl_wait();
    __shared__ float tile[32][33];
    const int tap = blockIdx.z;
    const int n0 = blockIdx.x * 32, k0 = blockIdx.y * 32;       // n: output channel, k: input channel
    const float* wt = w + (size_t)tap * Cin * Cout;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int k = k0 + threadIdx.y + 8 * r, n = n0 + threadIdx.x;
        const float v = (k < Cin && n < Cout) ? wt[(size_t)k * Cout + n] : 0.f;
        tile[threadIdx.y + 8 * r][threadIdx.x] = v;
        if (dx != nullptr && k < Cin_p && n < Cout_p) dx[((size_t)tap * Cin_p + k) * Cout_p + n] = static_cast<OutT>(v);
    }
    if (fwd == nullptr) return;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int n = n0 + threadIdx.y + 8 * r, k = k0 + threadIdx.x;
        if (n < Cout_p && k < Cin_p) fwd[((size_t)tap * Cout_p + n) * Cin_p + k] = static_cast<OutT>(tile[threadIdx.x][threadIdx.y + 8 * r]);
    }
}

template <typename OutT>
static int launch_filter_shadows(const float* w, OutT* fwd, OutT* dx, int taps, int Cin, int Cout, int Cin_p, int Cout_p,
                                 cudaStream_t st) {
    const dim3 grid((unsigned)ceil_div(Cout_p, 32), (unsigned)ceil_div(Cin_p, 32), (unsigned)taps);
    launch(filter_shadow_tiled_kernel<OutT>, grid, dim3(32, 8), 0, st, w, fwd, dx, Cin, Cout, Cin_p, Cout_p);
    count_launch();
    return check_launch("filter_shadow_tiled_kernel");
}

// ====================================================================================== host side
struct TcPlan {
    bool tf32;
    int Ho, Wo, taps;
    int elt;          // operand element size
    int KC;           // elements per 128-byte block
    int Cin_p, Cout_p;
    // workspace offsets (bytes)
    size_t off_xsh, off_dysh, off_wf, off_wd, off_part, off_dbpart, total;
    // dW decomposition
    int dw_nb, dw_nt, dw_cblocks, dw_U, dw_MG, dw_gpc, dw_ngc, dw_ntn, dw_splits;
    bool dw_pair;     // per-tap dW kernel on CTA pairs: dw_MG / dw_gpc / dw_ntn count pair groups and pair column tiles
    bool dw_small;    // operands in L2: the per-tap dW kernel with the decomposition chosen for few partials
    int dw_halo_splits;   // most splits the halo dW kernel may write (sizes the partial buffer with dw_splits)
    int db_blocks, db_rows_max;
    PixelTiling til_out;   // tiles over output pixels (forward, dW)
    PixelTiling til_in;    // tiles over input pixels (dX)
};

static int round_up(int v, int m) { return (v + m - 1) / m * m; }

// SM count of the calling thread's current device (looked up once per device).
int num_sms() {
    static std::atomic<int> cache[AE_MAX_DEVICES];
    const int dev = current_device();
    int n = cache[dev].load(std::memory_order_relaxed);
    if (n <= 0) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cache[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

// A stand-in with the pair kernels' launch shape for the occupancy query below.
__global__ void __launch_bounds__(IGEMM_THREADS, 1) pair_probe_kernel() { pdl_wait(); }

bool cta_pairs_available() {
    static std::atomic<int> cache[AE_MAX_DEVICES];       // 0 = not asked yet, 1 = yes, 2 = no
    const int dev = current_device();
    int v = cache[dev].load(std::memory_order_relaxed);
    if (v == 0) {
        v = 2;
        const int smem = IgemmCfg<256, true>::SMEM_BYTES;
        if (cudaFuncSetAttribute(pair_probe_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess) {
            cudaLaunchConfig_t cfg;
            memset(&cfg, 0, sizeof(cfg));
            cfg.gridDim = dim3(2 * (num_sms() / 2), 1, 1);
            cfg.blockDim = dim3(IGEMM_THREADS, 1, 1);
            cfg.dynamicSmemBytes = smem;
            cudaLaunchAttribute attr;
            attr.id = cudaLaunchAttributeClusterDimension;
            attr.val.clusterDim.x = 2;
            attr.val.clusterDim.y = 1;
            attr.val.clusterDim.z = 1;
            cfg.attrs = &attr;
            cfg.numAttrs = 1;
            int clusters = 0;
            if (cudaOccupancyMaxActiveClusters(&clusters, pair_probe_kernel, &cfg) == cudaSuccess && clusters >= num_sms() / 2) v = 1;
        }
        (void)cudaGetLastError();
        cache[dev].store(v, std::memory_order_relaxed);
    }
    return v == 1;
}

static TcPlan compute_plan(const AetherConvDesc& d) {
    TcPlan pl{};
    pl.tf32 = (d.math_mode == AETHER_MATH_TF32);
    conv_out_hw(d, pl.Ho, pl.Wo);
    pl.taps = d.fH * d.fW;
    pl.elt = pl.tf32 ? 4 : 2;
    pl.KC = 128 / pl.elt;
    pl.Cin_p = round_up(d.Cin, pl.KC);
    pl.Cout_p = round_up(d.Cout, pl.KC);
    pl.til_out = choose_tiling(d.S, pl.Ho, pl.Wo);
    pl.til_in = choose_tiling(d.S, d.H, d.W);
    // dW decomposition
    const int UC = pl.KC;
    const int MB = 128 / UC;
    if (pl.tf32) pl.dw_nb = (pl.Cout_p % 64 == 0) ? 2 : 1;
    else pl.dw_nb = (pl.Cout_p % 128 == 0) ? 2 : 1;
    pl.dw_nt = pl.dw_nb * UC;
    pl.dw_cblocks = pl.Cin_p / UC;
    pl.dw_U = pl.taps * pl.dw_cblocks;
    const long long ptiles = pl.til_out.total();
    auto decompose = [&](int pf, int max_gpc) {       // pf CTAs per M group and column tile, groups of a CTA (0: as many as TMEM holds); returns the split count
        pl.dw_MG = ceil_div(pl.dw_U, MB * pf);
        if (max_gpc == 0) max_gpc = 512 / (pl.dw_nt * pf);
        pl.dw_ngc = ceil_div(pl.dw_MG, max_gpc);
        pl.dw_gpc = ceil_div(pl.dw_MG, pl.dw_ngc);
        pl.dw_ngc = ceil_div(pl.dw_MG, pl.dw_gpc);
        pl.dw_ntn = pl.Cout_p / (pl.dw_nt * pf);
        long long want = (num_sms() / pf) / (pl.dw_ngc * pl.dw_ntn);
        if (want > ptiles) want = ptiles;
        return (int)want;
    };
    // Small layers, whose operands stay in L2: the products are cheap, what counts is how many CTAs share them and how many
    // partials they leave.  One M group per CTA and few splits against many groups and as many splits as SMs: estimated
    // per candidate from what a stage (64 KB from L2), an accumulator's store and the partials' way through L2 take.
    // (128 images 8x8 64->128: 128 CTAs x 64 partials of 295 KB -> 29 partials; Dense 784->128 at batch 128: 2 CTAs -> 7.)
    auto decompose_small = [&]() {
        pl.dw_MG = ceil_div(pl.dw_U, MB);
        pl.dw_ntn = pl.Cout_p / pl.dw_nt;
        const double t_box = 0.45 / 4.0, t_store = 0.5;                         // a box of 16 KB from L2; an accumulator's store
        const double dw_us = 2.0 * pl.dw_U * UC * pl.Cout_p * 4.0 / 4e6;        // a partial written and read at 4 TB/s
        const int max_gpc = 512 / pl.dw_nt;
        double best = 1e30;
        int best_gpc = 1, best_splits = 1;
        for (int g = 1; g <= max_gpc && g <= pl.dw_MG; ++g) {
            const long long cols = 1LL * ceil_div(pl.dw_MG, g) * pl.dw_ntn;
            for (long long s = 1; s <= ptiles && s * cols <= num_sms(); ++s) {
                const double cost = (double)((ptiles + s - 1) / s) * (g * MB + pl.dw_nb) * t_box + g * t_store + (s > 1 ? 1.5 + s * dw_us : 0.0);
                if (cost < best - 1e-9) { best = cost; best_gpc = g; best_splits = (int)s; }
            }
        }
        if (best == 1e30) return 0;
        pl.dw_gpc = best_gpc;
        pl.dw_ngc = ceil_div(pl.dw_MG, best_gpc);
        return best_splits;
    };
    // pairs: the channel counts must fill 256 rows and two column halves, and every pair needs a few pixel tiles
    pl.dw_halo_splits = decompose(1, 0);
    if (pl.dw_halo_splits < 1) pl.dw_halo_splits = 1;
    pl.dw_splits = pl.dw_halo_splits;
    pl.dw_pair = pl.dw_nb == 2 && pl.Cout_p % (2 * pl.dw_nt) == 0 && pl.dw_U >= 2 * MB && cta_pairs_available();
    if (pl.dw_pair) {
        const int ps = decompose(2, 0);
        if (ps < 1 || ptiles < 4LL * ps) {
            pl.dw_pair = false;
            decompose(1, 0);
        } else {
            // M groups per CTA: the count is chosen by how evenly the groups and pixels divide and by the partials (written, and read again).  In bf16 a tile of
            // pixels takes some 0.72 us for each, whether or not they share dy's half; in TF32, bound by the operands' way, sharing counts, more so where rows
            // of channels are no multiple of 128 bytes.  One group instead of two, dW with its reduction, us: 256 x 8x8 256->256 28.8 -> 21.9, 512 x 16x16
            // 128->256 68.7 -> 61.5, 4096 x 8x8 256->512 414 -> 376, 64 x 9x9 256->256 5x5 33 -> 28, TF32 256 x 16x16 128->128 48.2 -> 43.9; but TF32 81 x 104x12
            // 148->236 271 with one, 209 with three, 31 x 81x28 292->236 5x5 713 / 566.  Over 1659 shapes in bf16 and 2437 in TF32 the choice is at most 5 and 18 % behind
            // the best count, 0.1 and 0.8 % in the mean; with bf16's figure TF32 is up to 52 and 5.1 %, with as many groups as TMEM holds bf16 up to 84 %, TF32 63 %.
            const double dw_us = 2.0 * pl.dw_U * UC * pl.Cout_p * 4.0 / 4e6;        // as below
            const double tile = !pl.tf32 ? 0.0 : d.Cout % UC ? 0.13 : 0.07, group = !pl.tf32 ? 0.72 : d.Cin % UC ? 0.52 : 0.45;
            double best = 1e30;
            int gpc = 0;
            for (int g = 512 / (pl.dw_nt * 2); g >= 1; --g) {
                const int splits = decompose(2, g);
                if (splits < 1) continue;
                const double cost = (double)((ptiles + splits - 1) / splits) * (tile + pl.dw_gpc * group) + (pl.tf32 ? 0.2 : 1.0) * pl.dw_gpc +
                                    (splits == 1 ? 0.0 : pl.tf32 ? 1.9 + 0.42 * splits * dw_us : splits * dw_us);
                if (cost < best - 1e-9) { best = cost; gpc = g; }
            }
            pl.dw_splits = decompose(2, gpc);
        }
    }
    pl.dw_small = false;
    if (!pl.dw_pair && (1LL * d.S * d.H * d.W * pl.Cin_p + 1LL * d.S * pl.Ho * pl.Wo * pl.Cout_p) * pl.elt <= (32LL << 20)) {
        const int s = decompose_small();
        if (s > 0) {
            pl.dw_splits = s;
            pl.dw_small = true;
        } else {
            decompose(1, 0);
        }
    }
    const long long out_rows = 1LL * d.S * pl.Ho * pl.Wo;
    pl.db_blocks = (int)(out_rows < 4LL * num_sms() * 64 ? (out_rows + 63) / 64 : 4LL * num_sms());
    if (pl.db_blocks < 1) pl.db_blocks = 1;

    // workspace
    size_t off = 0;
    auto take = [&](size_t bytes) { size_t o = off; off = align_up(off + bytes, 1024); return o; };
    const size_t in_rows = (size_t)d.S * d.H * d.W;
    // the filter operands first: their place does not depend on the batch size, so they stay valid across batches
    pl.off_wf = take((size_t)pl.taps * pl.Cout_p * pl.Cin_p * pl.elt);
    pl.off_wd = take(pl.tf32 ? 0 : (size_t)pl.taps * pl.Cin_p * pl.Cout_p * pl.elt);
    pl.off_xsh = take(pl.tf32 ? 0 : in_rows * pl.Cin_p * 2);
    pl.off_dysh = take(pl.tf32 ? 0 : (size_t)out_rows * pl.Cout_p * 2);
    int part_splits = pl.dw_splits > pl.dw_halo_splits ? pl.dw_splits : pl.dw_halo_splits;
    if (!pl.tf32) {
        const int rs = rows_dw_max_splits(pl.Cin_p, pl.Cout_p, pl.Ho, pl.Wo, d.S, d.fH, d.fW);
        if (rs > part_splits) part_splits = rs;
    }
    pl.off_part = take((size_t)part_splits * pl.dw_U * UC * pl.Cout_p * 4);
    // rows of per-block column sums of dy: the cast pass writes db_blocks of them; a producer of dy that hands its own
    // in (aether_conv2d_operand_layout) may use up to db_rows_max
    pl.db_rows_max = pl.db_blocks > 8 * num_sms() ? pl.db_blocks : 8 * num_sms();
    pl.off_dbpart = take((size_t)pl.db_rows_max * d.Cout * 4);
    pl.total = off;
    return pl;
}

static const TcPlan& make_plan(const AetherConvDesc& d) { return cached_plan<TcPlan, compute_plan>(d); }

bool tc_conv_eligible(const AetherConvDesc& d) {
    if (d.math_mode != AETHER_MATH_BF16 && d.math_mode != AETHER_MATH_TF32) return false;
    if (d.sH != 1 || d.sW != 1) return false;
    if (d.Cin % 4 || d.Cout % 4) return false;           // 16-byte rows for the fp32 tensor maps
    if (d.Cin < 16 || d.Cout < 16) return false;         // tiny channel counts: the CUDA-core kernel is used
    if (d.fH * d.fW > 64) return false;
    int Ho, Wo;
    conv_out_hw(d, Ho, Wo);
    if (Ho < 1 || Wo < 1) return false;
    return true;
}

size_t tc_conv_workspace_bytes(const AetherConvDesc& d) { return make_plan(d).total; }

bool tc_conv_operand_layout(const AetherConvDesc& d, AetherOperandLayout* out) {
    if (!tc_conv_eligible(d) || d.math_mode != AETHER_MATH_BF16) return false;
    const TcPlan& pl = make_plan(d);
    out->x_copy_offset = pl.off_xsh;
    out->x_copy_ld = pl.Cin_p;
    out->dy_copy_offset = pl.off_dysh;
    out->dy_copy_ld = pl.Cout_p;
    out->dy_colsum_offset = pl.off_dbpart;
    out->dy_colsum_rows_max = pl.db_rows_max;
    return true;
}

// CTAs of the per-tap kernel.  With statistics the grid is a multiple of the number of column tiles, so that a
// CTA (tiles blockIdx.x + k * grid, column tile = tile % n_tiles_n) keeps one column tile throughout.
static int igemm_grid(long long m_tiles, int n_tiles_n, bool stats) {
    const long long total = m_tiles * n_tiles_n;
    int grid = (int)(total < num_sms() ? total : num_sms());
    if (stats && grid > n_tiles_n) grid -= grid % n_tiles_n;
    return grid;
}

// CTA pairs are used for 256- and 128-wide column tiles where there is enough work to give every pair of SMs at
// least two units.  Measured on B200 (batch 4096, bf16, single CTAs -> pairs): 16x16 128->256 forward 0.544 -> 0.461 ms
// and its dX (128 columns) 0.663 -> 0.597 ms, 8x8 256->512 forward 0.451 -> 0.406 ms and its dX 0.415 -> 0.383 ms.
// With one K chunk per stage the 128-column pair was SLOWER than single CTAs (0.709 ms): the one issuing thread then
// has 256 tensor clocks per stage for a barrier wait, four MMAs and two commits; two chunks per stage fixed that
// and also gave the 256-column pair 3-4 %.
static bool igemm_use_pairs(long long m_tiles, int nt, int n_tiles_n) {
    return (nt == 256 || nt == 192 || nt == 128) && (m_tiles + 1) / 2 * n_tiles_n >= 2LL * (num_sms() / 2) && cta_pairs_available();
}
static int igemm_pair_grid(long long m_tiles, int n_tiles_n, bool stats) {
    const long long units = (m_tiles + 1) / 2 * n_tiles_n;
    int pairs = (int)(units < num_sms() / 2 ? units : num_sms() / 2);
    if (stats && pairs > n_tiles_n) pairs -= pairs % n_tiles_n;
    return 2 * pairs;
}

// Column tile: the one whose rounds of units are through first.  What a 128-byte chunk of K takes, in clocks, is its operands' way from L2 (128 rows of
// pixels and the filter rows'); a unit's columns are stored while the next one's products run, so the longer of both counts, and a little of the other.  A tile
// that overhangs the channels costs what it copies, several tiles copy the pixels again.  The figures are fitted to every width's times over 1265 shapes of one
// and nine taps in both modes (K 16 to 2304, 64 to 3256 columns, 100 to 128000 rows): the choice is within 7 % of the fastest width everywhere, 0.2 % in the mean.
// (Without the stores, 3.3 %, up to 53 %: 1364 x 112->3256 15.3 us where 7.9 are there; widths that divide the channels only, 3.9 % in bf16, 9.7 % in TF32.  Before /
// now, us: bf16 256 x 8x8 256->192 forward 22.0 / 13.6, 192->160 17.6 / 11.2; TF32 150 x 16x16 160->96 54 / 29.  Few tiles are narrow: 128 rows of a Dense layer
// 2048 -> 256 15.7 in one tile, 12.3 in eight.)
static int pick_nt(int n_padded, long long m_tiles, int kiters, bool pairs = true, double* clocks = nullptr) {
    static const int widths[6] = {256, 192, 128, 96, 64, 32};
    const int sms = num_sms();
    const bool short_one = m_tiles * ceil_div(n_padded, 32) <= sms;   // (one round of the shortest)
    if (short_one && !clocks) return 32;
    int best = 32;
    double best_cost = 1e300;
    for (int nt : widths) {
        if (short_one && nt > 32) continue;
        const int cols = ceil_div(n_padded, nt);
        if (cols > 1 && nt > 128 && n_padded % nt) continue;          // (a filter tile reads on into the next tap's rows, a wide one by much)
        const bool pair = pairs && nt >= 128 && igemm_use_pairs(m_tiles, nt, cols);
        const long long units = pair ? (m_tiles + 1) / 2 * cols : m_tiles * cols, slots = pair ? sms / 2 : sms;
        const double mma = kiters * (170.0 + (pair ? 0.95 : 1.4) * nt), store = pair ? 1900.0 + 16.0 * nt : 400.0 + 11.0 * nt;
        const double cost = (double)((units + slots - 1) / slots) * (mma > store ? mma : store) + 0.4 * (mma > store ? store : mma);
        if (cost < best_cost - 1e-9) { best_cost = cost; best = nt; }
    }
    if (clocks) *clocks = best_cost;
    return best;
}
double per_tap_clocks(int n_padded, long long m_tiles, int kiters) {
    double c;
    pick_nt(n_padded, m_tiles, kiters, true, &c);
    return c;
}

template <bool TF32, int NT, bool STATS, bool PAIR, bool ACT = false, int RB = 128, bool POOLED = false, bool SPLIT = false>
static int launch_igemm_k(const IgemmParams& p, cudaStream_t st) {
    using Cfg = IgemmCfg<NT, PAIR, RB>;
    constexpr int SMEM = Cfg::SMEM_BYTES + (SPLIT ? IGEMM_SPLIT_BYTES : 0);
    static PerDeviceSmem configured;
    const auto kernel = igemm_conv_kernel<TF32, NT, STATS, PAIR, ACT, RB, POOLED, SPLIT>;
    if (int rc = ensure_dynamic_smem(kernel, SMEM, configured, "igemm_conv")) return rc;
    const long long m_tiles = 1LL * p.tiles_w * p.tiles_h * p.tiles_n;
    const int grid = PAIR ? igemm_pair_grid(m_tiles, p.n_tiles_n, STATS) : igemm_grid(m_tiles, p.n_tiles_n, STATS);
    if (STATS && (grid / (PAIR ? 2 : 1)) % p.n_tiles_n)
        return set_error(AE_UNSUPPORTED, "conv forward statistics: %d column tiles on %d CTAs", p.n_tiles_n, grid);
    const int pk = p.sgn > 0 ? PK_IGEMM_FWD : PK_IGEMM_DX;
    prof_begin(pk, st);
    if (PAIR) {
        launch_cluster(kernel, 2, grid, IGEMM_THREADS, SMEM, st, p);
    } else if (SPLIT) {
        launch_cluster(kernel, p.splits, (unsigned)(m_tiles * p.n_tiles_n * p.splits), IGEMM_THREADS, SMEM, st, p);
    } else {
        launch(kernel, grid, IGEMM_THREADS, SMEM, st, p);
    }
    prof_end(pk, st);
    count_launch();
    return check_launch("igemm_conv_kernel");
}

template <bool TF32, int NT>
static int launch_igemm(const IgemmParams& p, bool pair, bool narrow, cudaStream_t st) {
    if constexpr (!TF32 && NT <= 128) {
        if (narrow) return p.stats ? launch_igemm_k<false, NT, true, false, false, 64>(p, st) : launch_igemm_k<false, NT, false, false, false, 64>(p, st);
    }
    if constexpr (NT == 256 || NT == 192 || NT == 128) {
        if (pair) return p.stats ? launch_igemm_k<TF32, NT, true, true>(p, st) : launch_igemm_k<TF32, NT, false, true>(p, st);
    }
    if constexpr (!TF32 && NT == 32) {
        if (p.splits > 1)
            return p.act.out ? launch_igemm_k<false, 32, false, false, true, 128, false, true>(p, st) : launch_igemm_k<false, 32, false, false, false, 128, false, true>(p, st);
    }
    if constexpr (!TF32) {
        if (p.act.out) return launch_igemm_k<TF32, NT, false, false, true>(p, st);
    }
    return p.stats ? launch_igemm_k<TF32, NT, true, false>(p, st) : launch_igemm_k<TF32, NT, false, false>(p, st);
}

template <bool TF32>
static int dispatch_igemm(IgemmParams& p, int nt, bool pair, bool narrow, cudaStream_t st) {
    switch (nt) {
        case 256: return launch_igemm<TF32, 256>(p, pair, narrow, st);
        case 192: return launch_igemm<TF32, 192>(p, pair, narrow, st);
        case 128: return launch_igemm<TF32, 128>(p, pair, narrow, st);
        case 96: return launch_igemm<TF32, 96>(p, false, narrow, st);
        case 64: return launch_igemm<TF32, 64>(p, false, narrow, st);
        default: return launch_igemm<TF32, 32>(p, false, narrow, st);
    }
}

template <int NT>
static int launch_igemm_pooled(const IgemmParams& p, bool narrow, cudaStream_t st) {
    if constexpr (NT <= 128) {
        if (narrow) return launch_igemm_k<false, NT, false, false, false, 64, true>(p, st);
    }
    return launch_igemm_k<false, NT, false, false, false, 128, true>(p, st);
}

// Clusters of `size` CTAs of the SPLIT kernel that this device runs at once (looked up once per device and size): a GPC takes whole clusters, and how many SMs it has
// differs from one GPC and one GPU to the next.  74, 33 and 15 clusters of two, four and eight where this was measured.
static int split_clusters(int size) {
    static std::atomic<int> cache[AE_MAX_DEVICES][4];        // by log2 of the size, plus one
    const int dev = current_device(), k = size == 2 ? 1 : size == 4 ? 2 : 3;
    const int held = cache[dev][k].load(std::memory_order_relaxed);
    if (held > 0) return held - 1;
    const auto kernel = igemm_conv_kernel<false, 32, false, false, false, 128, false, true>;
    constexpr int SMEM = IgemmCfg<32, false>::SMEM_BYTES + IGEMM_SPLIT_BYTES;
    int clusters = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) == cudaSuccess) {
        cudaLaunchConfig_t cfg;
        memset(&cfg, 0, sizeof(cfg));
        cfg.gridDim = dim3(size * num_sms(), 1, 1);
        cfg.blockDim = dim3(IGEMM_THREADS, 1, 1);
        cfg.dynamicSmemBytes = SMEM;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = size;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess) clusters = 0;
    }
    (void)cudaGetLastError();
    cache[dev][k].store(clusters + 1, std::memory_order_relaxed);
    return clusters;
}

// CTAs that share a tile's K chunks (SPLIT): as many as there are SMs for in one round of clusters, with four chunks each at least, where that takes out twenty chunks of a
// CTA (a chunk is 0.16 us, the exchange 1.5; 896 x 2048->256 by two, 16 chunks less, 8.9 / 9.0 us).  (us: 256 x 3136->128 11.8 / 7.8, 128 x 2048->256 9.3 / 7.5, 256 x
// 8192->1024 24 / 16.7; 512 x 3136->128, 16 tiles, 16.1 / 13.3 by four, 18.4 by eight in two rounds.)
static int k_splits(long long tiles, int kchunks) {
    if (kchunks < 23) return 1;
    const int room = num_sms() * 7 / 8;
    for (int s = 8; s > 1; s >>= 1)
        if (tiles * s <= room && kchunks >= 4 * s && kchunks - kchunks / s >= 20 && tiles <= split_clusters(s)) return s;
    return 1;
}

// Runs out[p, n] = sum_{tap,k} in[p (+/-) tap, k] * Wm[tap][n][k] (+ bias).
static int run_igemm(bool tf32, const void* in, int in_C, int in_H, int in_W, int S, const void* wmat, int w_inner,
                     int rows_per_tap, int taps, float* out, int out_C, int out_H, int out_W, const PixelTiling& til,
                     int n_padded, int fH, int fW, int sgn, int off_h, int off_w, int k_real, const float* bias, float* stats,
                     cudaStream_t st, const ActEpilogue* act = nullptr, bool* act_done = nullptr, const PoolEpilogue* pool = nullptr) {
    if (pool == nullptr) {   // wide images with a filter that fits in shared memory: halo-reuse kernel
        bool used = false;
        const int padT = sgn > 0 ? -off_h : fH - 1 - off_h;
        const int padL = sgn > 0 ? -off_w : fW - 1 - off_w;
        int rc0 = run_halo_igemm(tf32, in, in_C, in_H, in_W, S, wmat, w_inner, rows_per_tap, taps, out, out_C, out_H, out_W,
                                 halo_n(out_C, n_padded), n_padded, til.total(), fH, fW, padT, padL, sgn > 0 ? 0 : 1, k_real, bias, stats,
                                 sgn > 0 ? PK_IGEMM_FWD : PK_IGEMM_DX, st, &used);
        if (rc0 || used) return rc0;
    }
    IgemmParams p;
    memset(&p, 0, sizeof(p));
    const int elt = tf32 ? 4 : 2;
    const CUtensorMapDataType dt = tf32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const int nt = pick_nt(n_padded, til.total(), taps * ceil_div(in_C, 128 / elt), pool == nullptr);
    const bool pair = pool == nullptr && igemm_use_pairs(til.total(), nt, ceil_div(n_padded, nt));   // each CTA of a pair stages half the filter rows
    const bool narrow = !tf32 && !pair && k_real <= 32 && nt <= 128 && (act == nullptr || stats != nullptr);
    const int KC = narrow ? 32 : 128 / elt;
    const CUtensorMapSwizzle swz = narrow ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B;
    int rc;
    if ((rc = make_map_nhwc(&p.tm_in, in, dt, elt, in_C, in_W, in_H, S, KC, til.BW, til.BH, til.BN, swz))) return rc;
    if ((rc = make_map_2d(&p.tm_w, wmat, dt, elt, w_inner, 1LL * taps * rows_per_tap, KC, pair ? nt / 2 : nt, swz))) return rc;
    if ((reinterpret_cast<uintptr_t>(out) & 15u) || (out_C & 3))
        return set_error(AE_BAD_ARG, "conv output must be 16-byte aligned with a channel count that is a multiple of 4");
    p.out = out;
    p.bias = bias;
    p.stats = stats;
    if (act != nullptr && !tf32 && !pair && stats == nullptr) {
        p.act = *act;
        *act_done = true;
    }
    p.status = device_status_word();
    p.n_out = out_C;
    p.out_W = out_W; p.out_H = out_H; p.out_N = S;
    p.BW = til.BW; p.BH = til.BH; p.BN = til.BN; p.rows = til.rows;
    p.tiles_w = til.tiles_w; p.tiles_h = til.tiles_h; p.tiles_n = til.tiles_n;
    p.n_tiles_n = ceil_div(n_padded, nt);
    p.rows_per_tap = rows_per_tap;
    p.fH = fH; p.fW = fW; p.sgn = sgn; p.off_h = off_h; p.off_w = off_w;
    p.kchunks = narrow ? 1 : ceil_div(in_C, KC);
    p.last_ksteps = narrow ? ceil_div(k_real, 16) : last_ksteps(k_real, p.kchunks, KC);
    p.splits = nt == 32 && taps == 1 && !tf32 && !narrow && stats == nullptr ? k_splits(til.total() * p.n_tiles_n, p.kchunks) : 1;
    if (pool != nullptr) {
        p.pool = *pool;
        switch (nt) {
            case 256: return launch_igemm_pooled<256>(p, narrow, st);
            case 192: return launch_igemm_pooled<192>(p, narrow, st);
            case 128: return launch_igemm_pooled<128>(p, narrow, st);
            case 96: return launch_igemm_pooled<96>(p, narrow, st);
            case 64: return launch_igemm_pooled<64>(p, narrow, st);
            default: return launch_igemm_pooled<32>(p, narrow, st);
        }
    }
    return tf32 ? dispatch_igemm<true>(p, nt, pair, false, st) : dispatch_igemm<false>(p, nt, pair, narrow, st);
}

static int launch_cast(const float* src, __nv_bfloat16* dst, long long rows, int C, int Cp, float* colsum_part,
                       int colsum_blocks, cudaStream_t st) {
    prof_begin(PK_SHADOW, st);
    if (colsum_part) {
        const long long rpb = (rows + colsum_blocks - 1) / colsum_blocks;
        launch(cast_bf16_kernel<true>, colsum_blocks, 256, 0, st, src, dst, rows, C, Cp, colsum_part, rpb);
    } else {
        long long blocks = 8LL * num_sms();
        const int G = Cp / 8;
        const int planes = G >= 256 ? 1 : 256 / G;
        if (blocks * planes > rows) blocks = (rows + planes - 1) / planes;
        if (blocks < 1) blocks = 1;
        const long long rpb = (rows + blocks - 1) / blocks;
        launch(cast_bf16_kernel<false>, (int)blocks, 256, 0, st, src, dst, rows, C, Cp, nullptr, rpb);
    }
    prof_end(PK_SHADOW, st);
    count_launch();
    return check_launch("cast_bf16_kernel");
}

long long tc_conv_stats_blocks(const AetherConvDesc& d) {
    if (!tc_conv_eligible(d)) return 0;
    const TcPlan& pl = make_plan(d);
    const long long hb = halo_igemm_stats_blocks(pl.tf32, pl.tf32 ? d.Cin : pl.Cin_p, d.S, pl.taps, d.Cout, pl.Ho, pl.Wo,
                                                 halo_n(d.Cout, pl.Cout_p), pl.Cout_p, pl.til_out.total(), d.fH, d.fW);
    if (hb > 0) return hb;
    // per-tap kernel: two rows per CTA group (the CTAs of one set of pixel tiles)
    const int nt = pick_nt(pl.Cout_p, pl.til_out.total(), pl.taps * ceil_div(pl.tf32 ? d.Cin : pl.Cin_p, pl.KC));
    const int n_tiles_n = ceil_div(pl.Cout_p, nt);
    if (igemm_use_pairs(pl.til_out.total(), nt, n_tiles_n)) {       // one block group per CTA of a pair
        const int pairs = igemm_pair_grid(pl.til_out.total(), n_tiles_n, true) / 2;
        if (pairs % n_tiles_n) return 0;
        return 4LL * (pairs / n_tiles_n);
    }
    const int grid = igemm_grid(pl.til_out.total(), n_tiles_n, true);
    if (grid % n_tiles_n) return 0;
    return 2LL * (grid / n_tiles_n);
}

// Both filter operands (forward: transposed, dX: as stored) from one read of w.
int tc_conv_filter_copies(const AetherConvDesc& d, const float* w, void* ws, size_t ws_bytes, cudaStream_t st) {
    const TcPlan& pl = make_plan(d);
    if (ws_bytes < pl.total) return set_error(AE_BAD_ARG, "conv workspace too small: %zu < %zu", ws_bytes, pl.total);
    uint8_t* wsb = static_cast<uint8_t*>(ws);
    return launch_filter_shadows<__nv_bfloat16>(w, reinterpret_cast<__nv_bfloat16*>(wsb + pl.off_wf), reinterpret_cast<__nv_bfloat16*>(wsb + pl.off_wd),
                                                pl.taps, d.Cin, d.Cout, pl.Cin_p, pl.Cout_p, st);
}

int tc_conv_fwd(const AetherConvDesc& d, const float* x, const float* w, const float* b, float* y, float* stats, void* ws,
                size_t ws_bytes, int flags, cudaStream_t st, const ActEpilogue* act, bool* act_done) {
    const TcPlan& pl = make_plan(d);
    if (ws_bytes < pl.total || !ws) return set_error(AE_BAD_ARG, "conv workspace too small: %zu < %zu", ws_bytes, pl.total);
    uint8_t* wsb = static_cast<uint8_t*>(ws);
    int rc;
    if (pl.tf32) {
        float* wf = reinterpret_cast<float*>(wsb + pl.off_wf);
        if (!(flags & AETHER_CONV_W_COPY_READY) &&
            (rc = launch_filter_shadows<float>(w, wf, nullptr, pl.taps, d.Cin, d.Cout, pl.Cin_p, pl.Cout_p, st)))
            return rc;
        return run_igemm(true, x, d.Cin, d.H, d.W, d.S, wf, pl.Cin_p, pl.Cout_p, pl.taps, y, d.Cout, pl.Ho, pl.Wo,
                         pl.til_out, pl.Cout_p, d.fH, d.fW, +1, -d.padH, -d.padW, d.Cin, b, stats, st);
    }
    __nv_bfloat16* xsh = reinterpret_cast<__nv_bfloat16*>(wsb + pl.off_xsh);
    __nv_bfloat16* wf = reinterpret_cast<__nv_bfloat16*>(wsb + pl.off_wf);
    // the bf16 copy of x: handed in by the kernel that produced x, else made here
    if (!(flags & AETHER_CONV_X_COPY_READY) &&
        (rc = launch_cast(x, xsh, 1LL * d.S * d.H * d.W, d.Cin, pl.Cin_p, nullptr, 0, st)))
        return rc;
    // (a backward call that is told the weights have not changed since -- x_shadow_valid bit 1 -- reuses the second of them)
    if (!(flags & AETHER_CONV_W_COPY_READY) && (rc = tc_conv_filter_copies(d, w, ws, ws_bytes, st))) return rc;
    return run_igemm(false, xsh, pl.Cin_p, d.H, d.W, d.S, wf, pl.Cin_p, pl.Cout_p, pl.taps, y, d.Cout, pl.Ho, pl.Wo,
                     pl.til_out, pl.Cout_p, d.fH, d.fW, +1, -d.padH, -d.padW, d.Cin, b, stats, st, act, act_done);
}

template <bool TF32, int NB, bool PAIR>
static int launch_dw(const DwParams& p, int splits, int grid_y, cudaStream_t st) {
    using Cfg = DwCfg<TF32, NB>;
    static PerDeviceSmem configured;
    if (int rc = ensure_dynamic_smem(dw_conv_kernel<TF32, NB, PAIR>, Cfg::SMEM_BYTES, configured, "dw_conv")) return rc;
    prof_begin(PK_DW, st);
    if (PAIR) {
        launch_cluster(dw_conv_kernel<TF32, NB, PAIR>, 2, dim3(2 * splits, grid_y), DW_THREADS, Cfg::SMEM_BYTES, st, p);
    } else {
        launch(dw_conv_kernel<TF32, NB, PAIR>, dim3(splits, grid_y), DW_THREADS, Cfg::SMEM_BYTES, st, p);
    }
    prof_end(PK_DW, st);
    count_launch();
    return check_launch("dw_conv_kernel");
}

// Boxes of 2x2 windows: 8 or 16 pixels wide, an even number of rows high, several images once a box is as high as one.
static PixelTiling choose_pool_tiling(int S, int H, int W) {
    PixelTiling best{};
    long long best_tiles = -1;
    for (int bw = 16; bw >= 8; bw -= 8)
        for (int bh = 2; bh <= H && bw * bh <= 128; bh += 2) {
            int bn = bh < H ? 1 : 128 / (bw * bh);
            if (bn > S) bn = S;
            const long long t = 1LL * ceil_div(W, bw) * ceil_div(H, bh) * ceil_div(S, bn);
            if (best_tiles < 0 || t < best_tiles) {
                best_tiles = t;
                best = PixelTiling{bw, bh, bn, bw * bh * bn, ceil_div(W, bw), ceil_div(H, bh), ceil_div(S, bn)};
            }
        }
    return best;
}
bool tc_conv_pool_eligible(const AetherConvDesc& d) {
    int Ho, Wo;
    conv_out_hw(d, Ho, Wo);
    return tc_conv_eligible(d) && d.math_mode == AETHER_MATH_BF16 && Ho % 2 == 0 && Wo % 2 == 0 && d.Cout <= IGEMM_POOL_CHANNELS;
}
// Whether that is ahead of the convolution by itself, which may keep windows or run on pairs and whose boxes fit any image, and the pass over its output.  Clocks of the
// rounds on either side (pick_nt; a pooled unit stores more slowly), the pass 2700 and 0.55 a KB.  us, pooled / apart: 896 x 16x16 32->64 30.8 / 47, 900 x 16x16
// 128->256 77 / 117, 128 x 8x8 256->512 31 / 36; but 900 x 18x18 16->16 82 / 33, 900 x 10x10 512->1024 1430 / 767, 128 x 10x10 256->256 34 / 24, 900 x 4x4
// 256->256 42 / 32.  Over 726 shapes at most 39 % behind the faster way, 0.6 % in the mean; pooled everywhere 145 % and 9 %.
bool tc_conv_pool_faster(const AetherConvDesc& d) {
    if (!tc_conv_pool_eligible(d)) return false;
    const TcPlan& pl = make_plan(d);
    const int kiters = pl.taps * ceil_div(pl.Cin_p, pl.KC), sms = num_sms();
    const long long tiles = choose_pool_tiling(d.S, pl.Ho, pl.Wo).total();
    const int nt = pick_nt(pl.Cout_p, tiles, kiters, false);
    const double mma = kiters * (210.0 + 1.1 * nt), store = 550.0 + 34.0 * nt;
    const double one = (double)((tiles * ceil_div(pl.Cout_p, nt) + sms - 1) / sms) * (mma > store ? mma : store) + 0.4 * (mma > store ? store : mma);
    double two = halo_igemm_clocks(false, pl.Cin_p, d.S, pl.taps, d.Cout, pl.Ho, pl.Wo, halo_n(d.Cout, pl.Cout_p), pl.Cout_p, pl.til_out.total(), d.fH, d.fW);
    if (two == 0.0) two = per_tap_clocks(pl.Cout_p, pl.til_out.total(), kiters);
    return one < two + 2700.0 + 0.55e-3 * 4.0 * d.S * pl.Ho * pl.Wo * d.Cout;
}
int tc_conv_fwd_pool(const AetherConvDesc& d, const float* x, const float* w, const float* b, const PoolEpilogue& pool, void* ws, size_t ws_bytes, int flags,
                     cudaStream_t st) {
    const TcPlan& pl = make_plan(d);
    if (ws_bytes < pl.total || !ws) return set_error(AE_BAD_ARG, "conv workspace too small: %zu < %zu", ws_bytes, pl.total);
    uint8_t* wsb = static_cast<uint8_t*>(ws);
    __nv_bfloat16* xsh = reinterpret_cast<__nv_bfloat16*>(wsb + pl.off_xsh);
    int rc;
    if (!(flags & AETHER_CONV_X_COPY_READY) && (rc = launch_cast(x, xsh, 1LL * d.S * d.H * d.W, d.Cin, pl.Cin_p, nullptr, 0, st))) return rc;
    if (!(flags & AETHER_CONV_W_COPY_READY) && (rc = tc_conv_filter_copies(d, w, ws, ws_bytes, st))) return rc;
    // (the output itself is not written: its rows are told from rows outside the image by their addresses)
    return run_igemm(false, xsh, pl.Cin_p, d.H, d.W, d.S, wsb + pl.off_wf, pl.Cin_p, pl.Cout_p, pl.taps, pool.pooled, d.Cout, pl.Ho, pl.Wo,
                     choose_pool_tiling(d.S, pl.Ho, pl.Wo), pl.Cout_p, d.fH, d.fW, +1, -d.padH, -d.padW, d.Cin, b, nullptr, st, nullptr, nullptr, &pool);
}

int tc_conv_bwd(const AetherConvDesc& d, const float* x, const float* dy, const float* w, float* dx, float* dw,
                float* db, void* ws, size_t ws_bytes, int x_shadow_valid, int dy_colsum_rows, cudaStream_t st) {
    const TcPlan& pl = make_plan(d);
    if (ws_bytes < pl.total || !ws) return set_error(AE_BAD_ARG, "conv workspace too small: %zu < %zu", ws_bytes, pl.total);
    uint8_t* wsb = static_cast<uint8_t*>(ws);
    int rc;
    const long long out_rows = 1LL * d.S * pl.Ho * pl.Wo;
    const long long in_rows = 1LL * d.S * d.H * d.W;
    float* dbpart = reinterpret_cast<float*>(wsb + pl.off_dbpart);
    const void* x_op = x;
    const void* dy_op = dy;
    const bool w_shadow_valid = (x_shadow_valid & AETHER_CONV_W_COPY_READY) != 0;
    const bool dy_ready = (x_shadow_valid & AETHER_CONV_DY_COPY_READY) != 0 && !pl.tf32;
    x_shadow_valid &= AETHER_CONV_X_COPY_READY;
    int db_rows = pl.db_blocks;
    if (dy_ready) {
        if (dy_colsum_rows < 1 || dy_colsum_rows > pl.db_rows_max)
            return set_error(AE_BAD_ARG, "aether_conv2d_bwd_ex: dy_colsum_rows %d outside [1, %d]", dy_colsum_rows, pl.db_rows_max);
        db_rows = dy_colsum_rows;
    }

    // ---- shadows + dB
    if (pl.tf32) {
        if (db) {
            const long long rpb = (out_rows + pl.db_blocks - 1) / pl.db_blocks;
            launch(colsum_kernel, pl.db_blocks, 256, 0, st, dy, out_rows, d.Cout, dbpart, rpb);
            count_launch();
            if ((rc = check_launch("colsum_kernel"))) return rc;
        }
    } else {
        __nv_bfloat16* dysh = reinterpret_cast<__nv_bfloat16*>(wsb + pl.off_dysh);
        __nv_bfloat16* xsh = reinterpret_cast<__nv_bfloat16*>(wsb + pl.off_xsh);
        // the bf16 copy of dy and the column sums for dB: handed in by the kernel that produced dy, else made here
        if (!dy_ready && (rc = launch_cast(dy, dysh, out_rows, d.Cout, pl.Cout_p, dbpart, pl.db_blocks, st))) return rc;
        if (dw && !x_shadow_valid)
            if ((rc = launch_cast(x, xsh, in_rows, d.Cin, pl.Cin_p, nullptr, 0, st))) return rc;
        x_op = xsh;
        dy_op = dysh;
    }
    // ---- dX: gather over dy with the filter read as (rows = Cin, K = Cout)
    if (dx) {
        if (pl.tf32) {
            // the caller's (taps, Cin, Cout) array already is the K-major matrix needed here
            rc = run_igemm(true, dy, d.Cout, pl.Ho, pl.Wo, d.S, w, d.Cout, d.Cin, pl.taps, dx, d.Cin, d.H, d.W,
                           pl.til_in, pl.Cin_p, d.fH, d.fW, -1, d.padH, d.padW, d.Cout, nullptr, nullptr, st);
        } else {
            __nv_bfloat16* wd = reinterpret_cast<__nv_bfloat16*>(wsb + pl.off_wd);
            if (!w_shadow_valid &&
                (rc = launch_filter_shadows<__nv_bfloat16>(w, nullptr, wd, pl.taps, d.Cin, d.Cout, pl.Cin_p, pl.Cout_p, st)))
                return rc;
            rc = run_igemm(false, dy_op, pl.Cout_p, pl.Ho, pl.Wo, d.S, wd, pl.Cout_p, pl.Cin_p, pl.taps, dx, d.Cin, d.H,
                           d.W, pl.til_in, pl.Cin_p, d.fH, d.fW, -1, d.padH, d.padW, d.Cout, nullptr, nullptr, st);
        }
        if (rc) return rc;
    }

    // ---- dW: split over pixel tiles, fixed-order reduction of the partials
    bool dw_done = false, db_done = db == nullptr;
    auto reduce_dw = [&](const float* part, int splits, int tap_split, int splits2) {
        db_done = true;
        return dw_reduce(part, dw, splits, pl.dw_U, pl.KC, pl.Cout_p, pl.dw_cblocks, pl.taps, d.Cin, d.Cout, tap_split, splits2, dbpart,
                         db_rows, db, st);
    };
    // Which dW kernel (bf16).  The kernels that reuse a shared-memory window across the taps win on wide images, but for channel counts that fill
    // the per-tap kernel's pairs of CTAs (256 output channels; of 64 input channels every fourth group would be padding).  Measured on
    // B200, window kernel / pair kernel in us, 80 GFLOP: 256 -> 256 channels 12x12 73 / 60, 16x16 71 / 60, 24x24 74 / 63, 32x32 70 / 60, 64x64
    // 72 / 58; 128 -> 256 12x12 71 / 68, 16x16 70 / 69, 24x24 72 / 70, 32x32 69 / 70, 64x64 75 / 67; on single CTAs 128 -> 128 69-77 / 79-87, 192
    // -> 192 107-121 / 113-129, 64 -> 64 106-114 / 123-144.
    const bool per_tap_pairs = pl.dw_pair && (pl.Cin_p >= 128 || (pl.Wo >= 16 && pl.Wo <= 20));
    // Small layers take the per-tap kernel, too: the window kernels spread one strip per CTA over as many splits as there are
    // SMs, and the partials cost more than the products (128 images 16x16 32->64: 17 + 7 us against 9 + 4).
    if (dw && !pl.tf32 && !per_tap_pairs && !pl.dw_small) {   // wide images: halo-reuse kernel (every tap re-reads one shared-memory window)
        int splits = 0;
        float* part = reinterpret_cast<float*>(wsb + pl.off_part);
        int sa = 0, sb = 0, tap_split = 0;
        if ((rc = run_rows_dw(x_op, pl.Cin_p, d.H, d.W, d.S, dy_op, pl.Cout_p, pl.Ho, pl.Wo, d.fH, d.fW, d.padH, d.padW, part,
                              &sa, &sb, &tap_split, st, &dw_done)))
            return rc;
        if (dw_done) {
            if ((rc = reduce_dw(part, sa, tap_split, sb))) return rc;
        }
        if (!dw_done) {
            if ((rc = run_halo_dw(x_op, pl.Cin_p, d.H, d.W, d.S, dy_op, pl.Cout_p, pl.Ho, pl.Wo, d.fH, d.fW, d.padH, d.padW,
                                  part, pl.dw_halo_splits, &splits, st, &dw_done)))
                return rc;
            if (dw_done) {
                if ((rc = reduce_dw(part, splits, pl.taps, splits))) return rc;
            }
        }
    }
    if (dw && !dw_done) {
        DwParams p;
        memset(&p, 0, sizeof(p));
        const CUtensorMapDataType dt = pl.tf32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
        const PixelTiling& til = pl.til_out;
        const int xC = pl.tf32 ? d.Cin : pl.Cin_p;
        const int dyC = pl.tf32 ? d.Cout : pl.Cout_p;
        const CUtensorMapSwizzle swz = pl.tf32 ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B;
        if ((rc = make_map_nhwc(&p.tm_x, x_op, dt, pl.elt, xC, d.W, d.H, d.S, pl.KC, til.BW, til.BH, til.BN, swz)))
            return rc;
        if ((rc = make_map_nhwc(&p.tm_dy, dy_op, dt, pl.elt, dyC, pl.Wo, pl.Ho, d.S, pl.KC, til.BW, til.BH, til.BN, swz)))
            return rc;
        // One split and no padded channels: the partial buffer's layout [tap*Cin + c][Cout] IS the layout of dW, so
        // the kernel writes the gradient itself and no reduction pass follows (a Dense layer's 8192 x 1024 matrix).
        const bool direct = pl.dw_splits == 1 && pl.Cin_p == d.Cin && pl.Cout_p == d.Cout;
        p.part = direct ? dw : reinterpret_cast<float*>(wsb + pl.off_part);
        p.status = device_status_word();
        p.BW = til.BW; p.BH = til.BH; p.BN = til.BN; p.rows = til.rows;
        p.tiles_w = til.tiles_w; p.tiles_h = til.tiles_h; p.tiles_n = til.tiles_n;
        p.fH = d.fH; p.fW = d.fW; p.padH = d.padH; p.padW = d.padW;
        p.cblocks = pl.dw_cblocks; p.U = pl.dw_U; p.MG = pl.dw_MG; p.gpc = pl.dw_gpc;
        p.n_tiles_n = pl.dw_ntn; p.ldn = pl.Cout_p; p.Cin = d.Cin; p.Cout = d.Cout;
        const int gy = pl.dw_ngc * pl.dw_ntn;
        if (pl.dw_pair) rc = pl.tf32 ? launch_dw<true, 2, true>(p, pl.dw_splits, gy, st) : launch_dw<false, 2, true>(p, pl.dw_splits, gy, st);
        else if (pl.tf32) rc = (pl.dw_nb == 2) ? launch_dw<true, 2, false>(p, pl.dw_splits, gy, st) : launch_dw<true, 1, false>(p, pl.dw_splits, gy, st);
        else rc = (pl.dw_nb == 2) ? launch_dw<false, 2, false>(p, pl.dw_splits, gy, st) : launch_dw<false, 1, false>(p, pl.dw_splits, gy, st);
        if (rc) return rc;
        if (!direct) {
            if ((rc = reduce_dw(p.part, pl.dw_splits, pl.taps, pl.dw_splits))) return rc;
        }
    }
    if (!db_done) return colsum_finish(dbpart, db_rows, d.Cout, db, st);
    return AE_OK;
}

}  // namespace aether
