// First-layer convolution (1..4 input channels, K = fH*fW*Cin <= 64) on the tensor cores, bf16 mode.
//
//   y[p][d] = b[d] + sum_k col[p][k] * w[k][d]            (Conv_Layer.forward, CNN_classes_cupy.py:70-120)
//
// With 3 input channels a pixel's 12 bytes cannot be the inner extent of a TMA box and K = 27 is less than one
// 128-byte operand row, so the im2col rows are built by threads: producer warps gather the K input values of
// 128 output pixels (one pixel per thread, all of a row's loads in flight together), convert them to bf16 and write them
// as a K-major, 128-byte-swizzled operand tile (16-byte chunk c of row r is stored at chunk c ^ (r % 8)); the filter is
// laid out the same way once per CTA.  One thread issues K/16 (two for a 3x3 RGB filter) 128 x Cout x 16 MMAs per tile into
// one of up to four TMEM accumulators.  Epilogue teams of four warps (two; up to four that pool) take tiles in turn: a thread reads 32 columns of
// its accumulator row, adds the bias and writes them to a swizzled staging tile that TMA stores to global memory; the
// statistics the following Batch_Norm needs are summed from the staged tile, a column per lane, so neither the exchange of
// columns between lanes nor their reduction across lanes is left.  A tile costs about 1700 warp instructions at 32 filters
// (6900 when every value went through shuffles and 64-byte register stores), the layer is bound by the HBM write of its
// output.
#include <cuda_bf16.h>
#include <string.h>

#include <type_traits>

#include "common.cuh"
#include "sm100_ptx.cuh"
#include "pool_epilogue.cuh"
#include "stats_epilogue.cuh"
#include "tc_host.cuh"

namespace aether {

// Producer warps, in groups of four that build tiles in turn: three groups where nothing but the gathers of few output channels holds the
// kernel back (896 x 32x32 3->32 35 -> 29 us, 64 and 128 channels 1-4 %), two with statistics, whose epilogue is the longer
// chain (128 x 32x32 3->32 10.9 us, 12.0 with three), and for windows of more than 48 values, which a thread keeps in registers: three groups
// leave it 80 of those (84 bytes spilled; 512 x 32x32 1->64 7x7 33.7 us, 31.6 with two groups, 64 x 64x64 4->32 4x4 19.8 / 18.9).  The pooling epilogue is the
// longer chain, too: four teams beside two groups (three and three: 1800 x 28x28 1->32 51.6 us, 49.5 so), as far as there are accumulators for them.
__host__ __device__ static constexpr int ft_prod_warps(bool stats, int KP, bool pooled) { return stats || KP > 48 || pooled ? 8 : 12; }
__host__ __device__ static constexpr int ft_teams(bool pooled) { return pooled ? 4 : 2; }       // of four epilogue warps, at most
__host__ __device__ static constexpr int ft_threads(bool stats, int KP, bool pooled) { return 32 * (ft_prod_warps(stats, KP, pooled) + 1 + 4 * ft_teams(pooled)); }      // producers, MMA issuer, epilogue
static constexpr int FT_STAGE_BYTES = 128 * 128;                             // 128 pixel rows of 128 bytes
static constexpr int FT_TAIL = 2048;                                         // barriers, TMEM pointer, bias, tap table
__host__ __device__ static constexpr int ft_out_bytes(bool pooled) { return ft_teams(pooled) * 2 * FT_STAGE_BYTES; }      // two staging tiles (128 rows x 32 floats) per team

__device__ __forceinline__ void ft_umma(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc,
                                        uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 da, {%1, %4};\n\tmov.b64 db, {%2, %4};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(hi), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// ---- the im2col gather shared by the forward and the filter-gradient kernel.  A thread builds one operand row: the K input
// values of one output pixel.  All of a row's loads are independent and issued together (a row is one load latency; in
// pieces of eight values it was three or four of them, each behind a 64-bit division of the pixel index).  3x3 filters on
// 1 or 3 channels, the usual first layers, have their offsets at compile time (CIN = 1, 3): two instructions per value.
struct FirstTaps {                 // entry k of a row: element offset from the window's first value, filter row | column << 8
    int2 t[64];
};
__device__ __forceinline__ void first_fill_taps(FirstTaps& tab, int K, int Cin, int fW, int W) {
    for (int k = threadIdx.x; k < 64; k += blockDim.x) {
        const int kk = k < K ? k : 0;
        const int tap = kk / Cin, c = kk - tap * Cin;
        const int i = tap / fW, j = tap - i * fW;
        tab.t[k] = make_int2((i * W + j) * Cin + c, k < K ? i | (j << 8) : 0x1f1f);   // past K: bit 31 of the masks, never set
    }
}
struct FirstGeom {
    const float* x;
    int P;                         // output pixels
    int H, W, Cin, fH, fW, sH, sW, pH, pW, Ho, Wo;
};
// POOLED: `pixel` counts the pixels of 2x2 windows, a window's four in row-major order one after the other.
template <int KP, int CIN, bool POOLED = false>
__device__ __forceinline__ void first_gather(const FirstGeom& g, const FirstTaps& tab, long long pixel, float (&v)[KP]) {
    unsigned rows = 0u, cols = 0u;                       // bit i / j: filter row i / column j falls inside the image
    const float* base = g.x;
    if (pixel < g.P) {
        const unsigned Wc = (unsigned)g.Wo >> (POOLED ? 1 : 0), Hc = (unsigned)g.Ho >> (POOLED ? 1 : 0);
        const unsigned u = (unsigned)pixel >> (POOLED ? 2 : 0), k = (unsigned)pixel & 3u, r = u / Wc, n = r / Hc;
        const int wo = POOLED ? (int)(2u * (u - r * Wc) + (k & 1u)) : (int)(u - r * Wc), ho = POOLED ? (int)(2u * (r - n * Hc) + (k >> 1)) : (int)(r - n * Hc);
        const int w0 = wo * g.sW - g.pW, h0 = ho * g.sH - g.pH;
        base = g.x + (((long long)n * g.H + h0) * g.W + w0) * (CIN ? CIN : g.Cin);     // may lie before the image
        const int i0 = h0 < 0 ? -h0 : 0, i1 = min(g.fH, g.H - h0), j0 = w0 < 0 ? -w0 : 0, j1 = min(g.fW, g.W - w0);
        if (i1 > i0) rows = (0xffffffffu >> (32 - i1)) & ~((1u << i0) - 1u);           // filters of at most 31 x 31
        if (j1 > j0) cols = (0xffffffffu >> (32 - j1)) & ~((1u << j0) - 1u);
    }
    if constexpr (CIN > 0) {
        const long long pitch = (long long)g.W * CIN;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const float* row = base + i * pitch;
            const unsigned m = ((rows >> i) & 1u) ? cols : 0u;
#pragma unroll
            for (int j = 0; j < 3; ++j)
#pragma unroll
                for (int c = 0; c < CIN; ++c) v[(i * 3 + j) * CIN + c] = ((m >> j) & 1u) ? __ldg(row + j * CIN + c) : 0.f;
        }
#pragma unroll
        for (int k = 9 * CIN; k < KP; ++k) v[k] = 0.f;
    } else {
#pragma unroll
        for (int k = 0; k < KP; ++k) {
            const int2 t = tab.t[k];
            v[k] = ((rows >> (t.y & 31)) & (cols >> (t.y >> 8)) & 1u) ? __ldg(base + t.x) : 0.f;
        }
    }
}
template <int KP>
__device__ __forceinline__ void first_store_row(uint8_t* tile, int r, const float (&v)[KP]) {
#pragma unroll
    for (int ch = 0; ch < KP / 8; ++ch)
        *reinterpret_cast<uint4*>(tile + r * 128 + ((ch ^ (r & 7)) << 4)) =
            make_uint4(pack_bf16(v[8 * ch], v[8 * ch + 1]), pack_bf16(v[8 * ch + 2], v[8 * ch + 3]), pack_bf16(v[8 * ch + 4], v[8 * ch + 5]),
                       pack_bf16(v[8 * ch + 6], v[8 * ch + 7]));
}

struct FirstParams {
    CUtensorMap tm_y;    // output (Cout, P) fp32, box (32 channels, 128 pixels), 128-byte swizzle
    FirstGeom g;
    const float* w;      // (fH, fW, Cin, Cout) = [K][Cout]
    const float* bias;   // nullable
    float* stats;        // nullable: [2 * cta][3][Cout] (count, mean, M2) partials (stats_epilogue.cuh)
    int* status;
    int Cout, NT, K;
    int stages, ntiles;
    PoolEpilogue pool;   // POOLED only
};

// Statistics: a thread sums one column over 32 rows of a tile, as eight sums of four rows each that a fixed tree adds up,
// about the mean of the CTA's first tile (no cancellation where a channel's mean is far from zero).  Up to 128 channels the
// eight sums run on over the CTA's tiles, in shared memory, and the tree comes at the end.  The two epilogue teams take
// every other tile and add to the running sums in tile order: a team waits for the other's statistics of the tile before
// (turn barriers, one per team and 32-channel chunk) with the tile's values already in registers, so that the exclusive part
// is short.  (128 channels at 4096 x 32x32: 423 us with sums of each team's own, 617 with both teams on every tile, 512 so;
// the network's statistics then do not depend on how its tiles meet the teams.)
// Shared memory: 16 turn barriers; float4[chunks][4][128] running sums (S, S, Q, Q; up to 128 channels); float[chunks][3][128]
// (pivot, S, Q); float[256] rows of each thread.
static constexpr int FT_TURN_BYTES = 128;
static int ft_stats_bytes(int NT) {
    const int NC = NT / 32;
    return FT_TURN_BYTES + (NT <= 128 ? NC * 4 * 128 * 16 : 0) + NC * 3 * 128 * 4 + 256 * 4;
}
__device__ __forceinline__ float stats_tree(const float (&v)[8]) { return ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7])); }

// POOLED (inference): the epilogue applies the Batch_Norm behind the layer by its running statistics, the (leaky) ReLU behind that and a 2x2
// max pooling, and writes the pooled values and their bf16 operand copy only, a quarter of the pixels.  A tile is 32 windows, whose four pixels are
// four rows of the staged tile, which takes the sums as they are: a thread reads four channels of a window again and keeps their coefficients, the eight lanes of
// a window read whole lines of banks.  (us, with the operand copy, against the convolution and the pass over its output: 900 x 32x32 3->32 35.6 / 66.6, 784 x 32x32
// 3->128 72.6, 900 x 32x32 3->192 153 / 433 on two teams; with the activation before the staging, eight channels a thread and two teams the first 47.)
template <bool STATS, int KP, int CIN, bool POOLED = false>
__global__ void __launch_bounds__(ft_threads(STATS, KP, POOLED), 1) first_conv_kernel(const __grid_constant__ FirstParams p) {
    constexpr int FT_PROD_WARPS = ft_prod_warps(STATS, KP, POOLED), TEAMS = ft_teams(POOLED);
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gen_base = smem_raw + (smem_base - smem_u32(smem_raw));
    const int NT = p.NT, S = p.stages;
    const uint32_t sW = smem_base;                                  // filter: NT rows of 128 bytes
    const uint32_t sA = sW + (uint32_t)NT * 128u;                   // NT is a multiple of 32: stays 1024-byte aligned
    const uint32_t sOut = sA + (uint32_t)S * FT_STAGE_BYTES;
    const uint32_t sBar = sOut + ft_out_bytes(POOLED);
    auto full_bar = [&](int s) { return sBar + 8u * s; };
    auto empty_bar = [&](int s) { return sBar + 8u * (S + s); };
    auto tfull_bar = [&](int b) { return sBar + 8u * (2 * S + b); };
    auto tempty_bar = [&](int b) { return sBar + 8u * (2 * S + 4 + b); };
    const uint32_t sTmemPtr = sBar + 8u * (2 * S + 8);
    volatile uint32_t* tmem_ptr_generic = reinterpret_cast<volatile uint32_t*>(gen_base + (sTmemPtr - smem_base));
    float* bias_s = reinterpret_cast<float*>(gen_base + (sBar - smem_base) + 256);         // NT <= 256 floats
    FirstTaps& taps = *reinterpret_cast<FirstTaps*>(gen_base + (sBar - smem_base) + 256 + 1024);
    const uint32_t sTurn = sBar + FT_TAIL;                                                 // STATS only, see above
    auto turn_bar = [&](int team, int ch) { return sTurn + 8u * (team * 8 + ch); };
    const bool persist = NT <= 128;
    float4* run_s = reinterpret_cast<float4*>(gen_base + (sTurn - smem_base) + FT_TURN_BYTES);
    float* stat_s = reinterpret_cast<float*>(run_s + (persist ? (NT >> 5) * 4 * 128 : 0));
    float* rows_s = stat_s + (NT >> 5) * 3 * 128;
    float* scale_s = reinterpret_cast<float*>(gen_base + (sTurn - smem_base));             // POOLED: scale, then shift
    float* shift_s = scale_s + NT;

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    // Accumulators, and the teams that take tiles: never more of these than of those.  A team waits for the parity of its tile's round, which an accumulator
    // that is two rounds behind shows as well: a third team on two accumulators would read one that the first still waits for.
    const int NB = (4 * NT <= 512) ? 4 : (3 * NT <= 512) ? 3 : 2;
    const int teams = POOLED ? min(TEAMS, NB) : TEAMS;
    static_assert(POOLED || TEAMS <= 2, "no more teams than accumulators");
    const uint32_t need_cols = (uint32_t)(NB * NT);
    const uint32_t tmem_cols = (need_cols <= 128) ? 128u : (need_cols <= 256) ? 256u : 512u;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(full_bar(s), 128);
            mbar_init(empty_bar(s), 1);
        }
        for (int b = 0; b < 4; ++b) {
            mbar_init(tfull_bar(b), 1);
            mbar_init(tempty_bar(b), 4);
        }
        if (STATS)
            for (int b = 0; b < 16; ++b) mbar_init(sTurn + 8u * b, 4);
        mbar_fence_init();
        if (!POOLED) tma_prefetch_desc(&p.tm_y);
    }
    if (CIN == 0) first_fill_taps(taps, p.K, p.g.Cin, p.g.fW, p.g.W);
    if (warp == FT_PROD_WARPS) {
        tmem_alloc(sTmemPtr, tmem_cols);
        tmem_relinquish();
    }
    pdl_wait();                       // set-up done; from here on global memory is touched
    for (int i = threadIdx.x; i < NT; i += blockDim.x) bias_s[i] = (p.bias != nullptr && i < p.Cout) ? p.bias[i] : 0.f;
    if (POOLED)
        for (int i = threadIdx.x; i < NT; i += blockDim.x) pool_coefficients(p.pool, i, p.Cout, scale_s[i], shift_s[i]);
    // filter operand: row n = output channel, element k at byte (k/8 ^ n%8)*16 + (k%8)*2 of the row
    for (int it = threadIdx.x; it < NT * (KP / 8); it += blockDim.x) {
        const int ch = it / NT, n = it - ch * NT;                  // neighbouring threads read neighbouring output channels
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int k = ch * 8 + e;
            v[e] = (n < p.Cout && k < p.K) ? p.w[(size_t)k * p.Cout + n] : 0.f;
        }
        const uint4 q = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
        *reinterpret_cast<uint4*>(gen_base + (sW - smem_base) + n * 128 + ((ch ^ (n & 7)) << 4)) = q;
    }
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_ptr_generic;
    const int grid = (int)gridDim.x;

    if (warp < FT_PROD_WARPS) {
        // ------------------------------------------------------------------ producers
        constexpr int GROUPS = FT_PROD_WARPS / 4;
        uint8_t* tile_gen = gen_base + (sA - smem_base);
        const int grp = threadIdx.x >> 7, r = threadIdx.x & 127;
        float v[KP];
        int t = blockIdx.x + grp * grid;
        if (t < p.ntiles) first_gather<KP, CIN, POOLED>(p.g, taps, (long long)t * 128 + r, v);
        for (int it = grp; t < p.ntiles; it += GROUPS) {
            const int s = it % S;
            if (!mbar_wait(empty_bar(s), ((uint32_t)(it / S) & 1u) ^ 1u, p.status, DS_TIMEOUT_EMPTY)) break;
            first_store_row<KP>(tile_gen + s * FT_STAGE_BYTES, r, v);
            fence_proxy_async_smem();                               // generic-proxy writes -> visible to the tensor core
            mbar_arrive(full_bar(s));
            t += GROUPS * grid;                                     // the next tile's loads are in flight meanwhile
            if (t < p.ntiles) first_gather<KP, CIN, POOLED>(p.g, taps, (long long)t * 128 + r, v);
        }
    } else if (warp == FT_PROD_WARPS) {
        // ------------------------------------------------------------------ MMA issuer (one thread)
        if (elect_one()) {
            const uint32_t idesc = make_idesc(1u, 0u, 0u, 128u, (uint32_t)NT);
            const uint64_t proto = make_smem_desc(0, 16, 1024);
            const uint32_t hi = (uint32_t)(proto >> 32);
            const uint32_t lo_proto = (uint32_t)proto;
            const uint32_t w_lo = lo_proto + ((sW & 0x3FFFFu) >> 4);
            const uint32_t a_lo0 = lo_proto + ((sA & 0x3FFFFu) >> 4);
            constexpr int ksteps = KP / 16;
            int it = 0;
            for (int t = blockIdx.x; t < p.ntiles; t += grid, ++it) {
                const int s = it % S, buf = it % NB;
                if (!mbar_wait(tempty_bar(buf), ((uint32_t)(it / NB) & 1u) ^ 1u, p.status, DS_TIMEOUT_TMEM_EMPTY)) break;
                if (!mbar_wait(full_bar(s), (uint32_t)(it / S) & 1u, p.status, DS_TIMEOUT_FULL)) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(buf * NT);
                const uint32_t a_lo = a_lo0 + (uint32_t)s * (FT_STAGE_BYTES >> 4);
#pragma unroll
                for (int ks = 0; ks < ksteps; ++ks) ft_umma(d_tmem, a_lo + 2u * ks, w_lo + 2u * ks, hi, idesc, ks ? 1u : 0u);
                umma_commit(empty_bar(s));
                umma_commit(tfull_bar(buf));
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue
        const int et = threadIdx.x - 32 * (FT_PROD_WARPS + 1);       // 0 .. 128 * TEAMS - 1
        const int team = et >> 7, tt = et & 127;
        const int q = warp & 3;                                      // TMEM lane quarter this warp may access
        const int row = q * 32 + lane;                               // accumulator row of this thread
        const int NC = NT >> 5;
        // statistics: this thread sums column `lane` of every chunk over rows [32 * part, 32 * part + 32)
        const int part = tt >> 5;
        float st_rows = 0.f;
        uint8_t* out_gen = gen_base + (sOut - smem_base) + team * 2 * FT_STAGE_BYTES;
        const uint32_t out_u = sOut + (uint32_t)(team * 2 * FT_STAGE_BYTES);
        int cnt = 0, it = team;
        bool ok = true, in_turn = true;
        for (int t = team < teams ? blockIdx.x + team * grid : p.ntiles; t < p.ntiles && ok; t += teams * grid, it += teams) {
            const int buf = it % NB;
            bool mine = in_turn && mbar_wait(tfull_bar(buf), (uint32_t)(it / NB) & 1u, p.status, DS_TIMEOUT_TMEM_FULL);
            tc_fence_after();
            const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * NT);
            const int left = p.g.P - t * 128;                        // rows of this tile
            const int r0 = part * 32, nr = STATS ? max(0, min(32, left - r0)) : 0;
            for (int ch = 0; ch < NC; ++ch, ++cnt) {
                uint8_t* o = out_gen + (cnt & 1) * FT_STAGE_BYTES;
                if (mine) {
                    uint32_t v[32];
                    tmem_ld_32x32(taddr + ch * 32, v);
                    tmem_ld_wait();
                    if (ch == NC - 1) {                               // accumulator fully read by this warp
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(tempty_bar(buf));
                    }
#pragma unroll
                    for (int c4 = 0; c4 < 8; ++c4) {
                        float4 a = make_float4(__uint_as_float(v[4 * c4]), __uint_as_float(v[4 * c4 + 1]), __uint_as_float(v[4 * c4 + 2]), __uint_as_float(v[4 * c4 + 3]));
                        if (!POOLED) {                                // (POOLED: where they are read again)
                            const float4 b = *reinterpret_cast<const float4*>(bias_s + ch * 32 + 4 * c4);
                            a = make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
                        }
                        *reinterpret_cast<float4*>(o + row * 128 + ((c4 ^ (row & 7)) << 4)) = a;
                    }
                    if (!POOLED) fence_proxy_async_smem();
                }
                if (!POOLED && tt == 0) tma_store_wait_read<0>();        // the other staging tile is free again
                ok = named_bar_and(1 + team, 128, mine);              // the tile is staged; a failed wait ends the whole team
                if (!ok) break;
                if (POOLED) {
                    // four channels of two windows per thread, eight neighbours a window's 32 (who writes this staging tile again has passed the other one's
                    // barrier, as everyone who reads here has)
                    const int c4 = tt & 7, col = ch * 32 + 4 * c4;
                    const float4 bi = *reinterpret_cast<const float4*>(bias_s + col), sc = *reinterpret_cast<const float4*>(scale_s + col);
                    const float4 sh = *reinterpret_cast<const float4*>(shift_s + col);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int window = (tt >> 3) + 16 * h;
                        const long long at = (long long)t * 32 + window;
                        if (at * 4 >= p.g.P) break;
                        float4 m[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const int r = window * 4 + k;
                            const float4 a = *reinterpret_cast<const float4*>(o + r * 128 + ((c4 ^ (r & 7)) << 4));
                            m[k] = pool_activation(make_float4(a.x + bi.x, a.y + bi.y, a.z + bi.z, a.w + bi.w), sc, sh, p.pool.alpha);
                        }
                        pool_store(p.pool, at, col, p.Cout, pool_first_max(m[0], m[1], m[2], m[3]));
                        for (int pad = NT + 4 * c4; ch == NC - 1 && pad < p.pool.ld; pad += 32)       // (columns of padding behind the last chunk)
                            pool_store(p.pool, at, pad, p.Cout, make_float4(0.f, 0.f, 0.f, 0.f));
                    }
                } else if (tt == 0) {
                    tma_store_2d(&p.tm_y, out_u + (uint32_t)((cnt & 1) * FT_STAGE_BYTES), ch * 32, t * 128);
                    tma_store_commit();
                }
                if (STATS) {
                    const bool first = it == 0;                       // sets the pivots
                    const uint8_t* col = o + r0 * 128 + (lane & 3) * 4;
                    float val[32];                                    // (rows past the last are never added)
#pragma unroll
                    for (int r = 0; r < 32; ++r) val[r] = *reinterpret_cast<const float*>(col + r * 128 + (((lane >> 2) ^ (r & 7)) << 4));
                    if (!first)                                       // the other team has added the tile before
                        in_turn = in_turn && mbar_wait(turn_bar(team, ch), (uint32_t)((it >> 1) - (team == 0 ? 1 : 0)) & 1u, p.status, DS_TIMEOUT_TMEM_FULL);
                    if (in_turn && nr > 0) {
                        float* base = stat_s + ch * 3 * 128 + tt;
                        float4* run = run_s + ch * 4 * 128 + tt;
                        float s8[8], q8[8];
                        if (first) {                                  // the mean first, then the squares about it
#pragma unroll
                            for (int k = 0; k < 8; ++k) s8[k] = 0.f;
#pragma unroll
                            for (int r = 0; r < 32; ++r) s8[r & 7] += r < nr ? val[r] : 0.f;
                            const float mean = stats_tree(s8) * (1.f / (float)nr);
                            base[0] = isfinite(mean) ? mean : 0.f;        // (else every value would differ from it by no number)
                            base[128] = base[256] = 0.f;
                        }
                        const float npiv = -base[0];
                        if (persist && !first) {
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                *reinterpret_cast<float4*>(s8 + 4 * h) = run[h * 128];
                                *reinterpret_cast<float4*>(q8 + 4 * h) = run[(2 + h) * 128];
                            }
                        } else {
#pragma unroll
                            for (int k = 0; k < 8; ++k) s8[k] = q8[k] = 0.f;
                        }
                        auto add_rows = [&](auto all) {
#pragma unroll
                            for (int r = 0; r < 32; ++r)
                                if (decltype(all)::value || r < nr) {
                                    const float d = val[r] + npiv;
                                    s8[r & 7] += d;
                                    q8[r & 7] = fmaf(d, d, q8[r & 7]);
                                }
                        };
                        if (nr == 32) add_rows(std::true_type{});
                        else add_rows(std::false_type{});
                        if (!persist) {
                            base[128] += stats_tree(s8);
                            base[256] += stats_tree(q8);
                        }
                        if (persist) {
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                run[h * 128] = *reinterpret_cast<const float4*>(s8 + 4 * h);
                                run[(2 + h) * 128] = *reinterpret_cast<const float4*>(q8 + 4 * h);
                            }
                        }
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(turn_bar(team ^ 1, ch));
                }
            }
            st_rows += (float)nr;
        }
        if (!POOLED && tt == 0) tma_store_wait_all<0>();
        if (STATS) {
            // two rows per CTA (stats_epilogue.cuh): the four threads of a column merged in fixed order
            rows_s[et] = st_rows;
            named_bar_sync(3, 256);
            float* sp = p.stats + (size_t)blockIdx.x * 6 * p.Cout;
            for (int c = et; c < p.Cout; c += 256) {
                double N = 0.0, S = 0.0, Q = 0.0;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int th = k * 32 + (c & 31);
                    const float n = rows_s[th] + rows_s[128 + th];
                    if (n == 0.f) continue;
                    const float* base = stat_s + (c >> 5) * 3 * 128 + th;
                    float s = base[128], q = base[256];
                    if (persist) {
                        const float4* run = run_s + (c >> 5) * 4 * 128 + th;
                        float v[8];
                        *reinterpret_cast<float4*>(v) = run[0];
                        *reinterpret_cast<float4*>(v + 4) = run[128];
                        s += stats_tree(v);
                        *reinterpret_cast<float4*>(v) = run[256];
                        *reinterpret_cast<float4*>(v + 4) = run[384];
                        q += stats_tree(v);
                    }
                    const float m2 = fmaxf(q - s * (s / n), 0.f);
                    const double mean = (double)base[0] + (double)s / (double)n;       // (rounded once, with the sums of all rows)
                    N += n; S += n * mean; Q += m2 + n * mean * mean;
                }
                stats_store_rows(N, S, Q, sp, c, p.Cout);
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == FT_PROD_WARPS) {
        tc_fence_after();
        tmem_dealloc(tmem_base, tmem_cols);
    }
}

// ====================================================================================== filter / bias gradient
//   dw[k][d] = sum_p col[p][k] * dy[p][d],  db[d] = sum_p dy[p][d]            (Conv_Layer.backward, :132-134)
// as D[d][k] += dy^T[d][pixels] * col[pixels][k]: M = 128 output channels (two 64-channel chunks of an MN-major
// operand), N = K padded to 16, reduction over the 128 pixels of a tile in eight K=16 steps.  The producers build
// both operands: the col tile exactly as in the forward kernel (the same bytes serve as an MN-major B operand) and
// the dy tile converted from fp32 to bf16; they also keep the fp32 column sums of dy for db.  The accumulators stay
// in TMEM for the CTA's whole life; one partial per CTA, summed in fixed order by smallc_reduce_kernel.
struct FirstDwParams {
    FirstGeom g;
    const float* dy;
    float* part;         // [cta][K + 1][Cout]
    int* status;
    int Cout, K, KP;
    int dblocks;         // 128-channel blocks of dy
    long long P;
    int stages, ntiles, stage_bytes;
    int groups;          // producer groups (divides FD_NP; <= stages)
    // dy handed in as a bf16 copy [P][dy_ld] by the kernel that produced it (aether_conv2d_operand_layout): TMA brings
    // the tile in already in operand form, the producers only gather the col tile, and dB comes from the column sums
    // that arrived with the copy
    CUtensorMap tm_dy;   // (dy_ld, P), box (64 channels, 128 pixels), 128-byte swizzle
    int dy_bf16;
};

// Twelve producer warps: with one producer warp per scheduler every round of dy loads costs a full HBM round trip
// and the kernel ran at a third of the HBM rate; 384 threads cover a 128-pixel tile of dy in one or two rounds.
static constexpr int FD_PROD_WARPS = 12;
static constexpr int FD_NP = 32 * FD_PROD_WARPS;
// Producer groups, each building every groups-th tile.  At most as many groups as operand stages: a group that
// could run two phases ahead of a stage's barrier would pass its parity wait early.
static constexpr int FD_MAX_GROUPS = 3;
static constexpr int FD_ROWS = 6;                                            // dy rows per thread and round
static constexpr int FD_TAIL = 1024 + FD_NP * 8 * 4 + 1024;                  // barriers, k tables, dB staging
static constexpr int FD_THREADS = 32 * (FD_PROD_WARPS + 1 + 4);              // producers, MMA issuer, 4 epilogue warps

template <int KP, int CIN>
__global__ void __launch_bounds__(FD_THREADS, 1) first_dw_kernel(const __grid_constant__ FirstDwParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gen_base = smem_raw + (smem_base - smem_u32(smem_raw));
    const int S = p.stages;
    const uint32_t sBar = smem_base + (uint32_t)S * p.stage_bytes;           // stage: col tile, then 2*dblocks dy chunks
    auto full_bar = [&](int s) { return sBar + 8u * s; };
    auto empty_bar = [&](int s) { return sBar + 8u * (S + s); };
    const uint32_t done_bar = sBar + 8u * (2 * S);
    const uint32_t sTmemPtr = sBar + 8u * (2 * S + 1);
    volatile uint32_t* tmem_ptr_generic = reinterpret_cast<volatile uint32_t*>(gen_base + (sTmemPtr - smem_base));
    FirstTaps& taps = *reinterpret_cast<FirstTaps*>(gen_base + (sBar - smem_base) + 256);
    float* dbsum_s = reinterpret_cast<float*>(gen_base + (sBar - smem_base) + 1024);      // [producer threads][8]

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    const uint32_t tmem_cols = 128;                                          // dblocks (<= 2) x KP (<= 64) columns

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(full_bar(s), FD_NP / p.groups + (p.dy_bf16 ? 1 : 0));    // + the thread that posts the TMA bytes
            mbar_init(empty_bar(s), 1);
        }
        mbar_init(done_bar, 1);
        mbar_fence_init();
        if (p.dy_bf16) tma_prefetch_desc(&p.tm_dy);
    }
    if (CIN == 0) first_fill_taps(taps, p.K, p.g.Cin, p.g.fW, p.g.W);
    if (warp == FD_PROD_WARPS) {
        tmem_alloc(sTmemPtr, tmem_cols);
        tmem_relinquish();
    }
    pdl_wait();                       // set-up done; from here on global memory is touched
    tc_fence_before();
    __syncthreads();

    tc_fence_after();
    const uint32_t tmem_base = *tmem_ptr_generic;
    const int grid = (int)gridDim.x;
    const bool any = (int)blockIdx.x < p.ntiles;

    if (warp < FD_PROD_WARPS) {
        // ------------------------------------------------------------------ producers
        // Groups of warps build alternate tiles: while one group converts and gathers, the other groups' dy loads are
        // in flight (all twelve warps in lock step left the HBM pipe idle for two thirds of every tile).
        const int r = threadIdx.x;                                   // 0 .. FD_NP-1
        const int FD_GRP = FD_NP / p.groups;
        const int grp = r / FD_GRP, rg = r - grp * FD_GRP;
        const int C8 = p.Cout >> 3;                                  // 8-channel chunks of a dy row (power of two <= 32)
        const int my_chunk = rg & (C8 - 1);                          // fixed for this thread: FD_GRP % C8 == 0
        const int prow0 = rg / C8, prow_step = FD_GRP / C8;
        const int dchunks = p.dblocks * 16;                          // 8-channel chunks the operand holds (zero padded)
        float bs[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) bs[e] = 0.f;
        if (C8 < dchunks) {
            // fewer than 128 channels: the chunks past Cout of the M = 128 operand are zero and stay zero (nobody
            // writes them again); published to the tensor core before any producer arrives on a stage
            for (int i = r; i < S * p.stage_bytes / 16; i += FD_NP)
                reinterpret_cast<uint4*>(gen_base)[i] = make_uint4(0, 0, 0, 0);
            fence_proxy_async_smem();
            named_bar_sync(1, FD_NP);
        }
        int k = grp;                                                 // index of the tile among this CTA's tiles
        for (int t = blockIdx.x + grp * grid; t < p.ntiles; t += p.groups * grid, k += p.groups) {
            const int s = k % S;
            const uint32_t ph = (uint32_t)(k / S) & 1u;
            const long long pix0 = (long long)t * 128;
            if (!mbar_wait(empty_bar(s), ph ^ 1u, p.status, DS_TIMEOUT_EMPTY)) break;
            uint8_t* stage = gen_base + (size_t)s * p.stage_bytes;
            // dy tile first (the long-latency loads): rows = pixels, 64-channel chunks of 128 bytes; chunk region c64
            // starts at 16 KB * (1 + c64).  All loads of a round are issued before the first use.
            uint8_t* reg = stage + FT_STAGE_BYTES * (1 + (my_chunk >> 3));
            if (p.dy_bf16 && rg == 0) {
                // the tile of the bf16 copy: one box per 64-channel chunk, rows past the last pixel are zero filled
                const int real_chunks = (p.Cout + 63) >> 6;
                mbar_arrive_expect_tx(full_bar(s), (uint32_t)real_chunks * FT_STAGE_BYTES);
                for (int c64 = 0; c64 < real_chunks; ++c64)
                    tma_load_2d(smem_base + (uint32_t)s * p.stage_bytes + FT_STAGE_BYTES * (1 + c64), &p.tm_dy, full_bar(s),
                                c64 * 64, (int)pix0);
            }
            for (int pr0 = prow0; pr0 < 128 && !p.dy_bf16; pr0 += FD_ROWS * prow_step) {
                float4 a[FD_ROWS], b[FD_ROWS];
#pragma unroll
                for (int u = 0; u < FD_ROWS; ++u) {
                    const int pr = pr0 + u * prow_step;
                    const long long pp = pix0 + pr;
                    a[u] = b[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (pr < 128 && pp < p.P) {
                        const float4* src = reinterpret_cast<const float4*>(p.dy + (size_t)pp * p.Cout + my_chunk * 8);
                        a[u] = __ldcs(src);
                        b[u] = __ldcs(src + 1);
                    }
                }
#pragma unroll
                for (int u = 0; u < FD_ROWS; ++u) {
                    const int pr = pr0 + u * prow_step;
                    if (pr < 128) {
                        bs[0] += a[u].x; bs[1] += a[u].y; bs[2] += a[u].z; bs[3] += a[u].w;
                        bs[4] += b[u].x; bs[5] += b[u].y; bs[6] += b[u].z; bs[7] += b[u].w;
                        const uint4 q = make_uint4(pack_bf16(a[u].x, a[u].y), pack_bf16(a[u].z, a[u].w),
                                                   pack_bf16(b[u].x, b[u].y), pack_bf16(b[u].z, b[u].w));
                        *reinterpret_cast<uint4*>(reg + pr * 128 + (((my_chunk & 7) ^ (pr & 7)) << 4)) = q;
                    }
                }
            }
            // col tile: row = pixel of the tile (the forward kernel's operand, read here as MN-major B)
            for (int pr = rg; pr < 128; pr += FD_GRP) {
                float v[KP];
                first_gather<KP, CIN>(p.g, taps, pix0 + pr, v);
                first_store_row<KP>(stage, pr, v);
            }
            fence_proxy_async_smem();
            mbar_arrive(full_bar(s));
        }
        // db: fp32 column sums of this thread's 8 channels; threads with the same chunk are added in fixed order
#pragma unroll
        for (int e = 0; e < 8; ++e) dbsum_s[r * 8 + e] = bs[e];
        named_bar_sync(1, FD_NP);
        for (int c = r; c < p.Cout; c += FD_NP) {          // (all zero when dy came as a copy: dB is taken elsewhere)
            const int ck = c >> 3, e = c & 7;
            float tsum = 0.f;
            for (int th = ck; th < FD_NP; th += C8) tsum += dbsum_s[th * 8 + e];
            p.part[(size_t)blockIdx.x * (p.K + 1) * p.Cout + (size_t)p.K * p.Cout + c] = tsum;
        }
    } else if (warp == FD_PROD_WARPS) {
        // ------------------------------------------------------------------ MMA issuer
        const bool leader = elect_one();
        const uint32_t idesc = make_idesc(1u, 1u, 1u, 128u, (uint32_t)KP);      // A and B MN-major
        const uint32_t hi = (uint32_t)(make_smem_desc(0, 0, 1024) >> 32);          // SBO = 8 reduction rows
        const uint32_t a_lbo = ((uint32_t)FT_STAGE_BYTES >> 4) << 16;              // next 64-channel chunk of dy
        int s = 0;
        uint32_t ph = 0, acc = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < p.ntiles && ok; t += grid) {
            bool f_ok = mbar_wait_spin(full_bar(s), ph, p.status, DS_TIMEOUT_FULL);
            f_ok = __all_sync(0xffffffffu, f_ok);
            if (!f_ok) { ok = false; break; }
            tc_fence_after();
            const uint32_t st16 = ((smem_base + (uint32_t)s * p.stage_bytes) & 0x3FFFFu) >> 4;
            if (leader) {
                for (int db = 0; db < p.dblocks; ++db) {
                    const uint32_t a0 = st16 + ((uint32_t)FT_STAGE_BYTES >> 4) * (1u + 2u * db);
                    for (uint32_t ks = 0; ks < 8; ++ks)
                        asm volatile(
                            "{\n\t.reg .pred pp;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 pp, %5, 0;\n\t"
                            "mov.b64 da, {%1, %4};\n\tmov.b64 db, {%2, %4};\n\t"
                            "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, pp;\n\t}"
                            ::"r"(tmem_base + (uint32_t)(db * 64)), "r"((a0 + ks * 128u) | a_lbo), "r"(st16 + ks * 128u),
                              "r"(idesc), "r"(hi), "r"((ks | acc) ? 1u : 0u)
                            : "memory");
                }
                umma_commit(empty_bar(s));
            }
            acc = 1u;
            if (++s == S) { s = 0; ph ^= 1u; }
            __syncwarp();
        }
        if (leader) umma_commit(done_bar);
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ epilogue: one partial per CTA
        const int q = warp & 3;
        bool ok = true;
        if (any) ok = mbar_wait(done_bar, 0, p.status, DS_TIMEOUT_TMEM_FULL);
        tc_fence_after();
        if (ok) {
            float* out = p.part + (size_t)blockIdx.x * (p.K + 1) * p.Cout;
            for (int db = 0; db < p.dblocks; ++db) {
                const int d = db * 128 + q * 32 + lane;
                for (int cg = 0; cg < KP; cg += 32) {
                    uint32_t v[32];
                    if (any) {
                        tmem_ld_32x32(tmem_base + ((uint32_t)(q * 32) << 16) + db * 64 + cg, v);
                        tmem_ld_wait();
                    } else {
#pragma unroll
                        for (int k = 0; k < 32; ++k) v[k] = 0u;
                    }
                    if (d < p.Cout) {
#pragma unroll
                        for (int k = 0; k < 32; ++k)
                            if (cg + k < p.K) out[(size_t)(cg + k) * p.Cout + d] = __uint_as_float(v[k]);
                    }
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == FD_PROD_WARPS) {
        tc_fence_after();
        tmem_dealloc(tmem_base, tmem_cols);
    }
}

// ---------------------------------------------------------------------------------- host
static bool first_tc_shape(const AetherConvDesc& d, int& K, int& KP, int& NT, int& Ho, int& Wo) {
    if (d.math_mode != AETHER_MATH_BF16) return false;
    K = d.fH * d.fW * d.Cin;
    if (d.Cin > 4 || K > 64 || d.fH > 31 || d.fW > 31) return false;
    if (d.Cout % 4 || d.Cout < 16 || d.Cout > 256) return false;
    KP = (K + 15) / 16 * 16;
    NT = (d.Cout + 31) / 32 * 32;              // whole 32-column chunks
    conv_out_hw(d, Ho, Wo);
    if (Ho < 1 || Wo < 1) return false;
    const long long P = 1LL * d.S * Ho * Wo;
    return P < 0x7fffff00LL;                   // pixel indices and TMA coordinates are 32-bit
}

bool first_tc_eligible(const AetherConvDesc& d) {
    int K, KP, NT, Ho, Wo;
    return first_tc_shape(d, K, KP, NT, Ho, Wo);
}

static int first_tc_grid(long long ntiles) { return (int)(ntiles < num_sms() ? ntiles : num_sms()); }

long long first_tc_stats_blocks(const AetherConvDesc& d) {
    int K, KP, NT, Ho, Wo;
    if (!first_tc_shape(d, K, KP, NT, Ho, Wo)) return 0;
    const long long P = 1LL * d.S * Ho * Wo;
    return 2LL * first_tc_grid((P + 127) / 128);
}

static FirstGeom first_geom(const AetherConvDesc& d, const float* x, int Ho, int Wo) {
    return FirstGeom{x, (int)(1LL * d.S * Ho * Wo), d.H, d.W, d.Cin, d.fH, d.fW, d.sH, d.sW, d.padH, d.padW, Ho, Wo};
}
// Kernel variant: 3x3 filters on 1 or 3 channels at compile time, else the tap table at K padded to 16, 32, 48, 64.
static int first_variant(const AetherConvDesc& d, int KP) {
    if (d.fH == 3 && d.fW == 3 && d.Cin == 1) return 4;
    if (d.fH == 3 && d.fW == 3 && d.Cin == 3) return 5;
    return KP / 16 - 1;
}

int first_tc_fwd(const AetherConvDesc& d, const float* x, const float* w, const float* b, float* y, float* stats,
                 cudaStream_t st, const PoolEpilogue* pool) {
    int K, KP, NT, Ho, Wo;
    if (!first_tc_shape(d, K, KP, NT, Ho, Wo)) return set_error(AE_UNSUPPORTED, "first_tc_fwd: shape not supported");
    FirstParams p;
    memset(&p, 0, sizeof(p));
    p.g = first_geom(d, x, Ho, Wo);
    p.w = w; p.bias = b; p.stats = stats; p.status = device_status_word();
    p.Cout = d.Cout; p.NT = NT; p.K = K;
    p.ntiles = (p.g.P + 127) / 128;
    p.stages = pool ? 3 : 4;
    if (pool) p.pool = *pool;
    else if (int rc = make_map_2d(&p.tm_y, y, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, d.Cout, p.g.P, 32, 128)) return rc;
    const int stat_bytes = stats ? ft_stats_bytes(NT) : pool ? NT * 8 : 0;
    const int smem = 1024 + NT * 128 + p.stages * FT_STAGE_BYTES + ft_out_bytes(pool != nullptr) + FT_TAIL + stat_bytes;
    using KernelFn = void (*)(const FirstParams);
    static const KernelFn kernels[3][6] = {{first_conv_kernel<false, 16, 0>, first_conv_kernel<false, 32, 0>, first_conv_kernel<false, 48, 0>,
                                            first_conv_kernel<false, 64, 0>, first_conv_kernel<false, 16, 1>, first_conv_kernel<false, 32, 3>},
                                           {first_conv_kernel<true, 16, 0>, first_conv_kernel<true, 32, 0>, first_conv_kernel<true, 48, 0>,
                                            first_conv_kernel<true, 64, 0>, first_conv_kernel<true, 16, 1>, first_conv_kernel<true, 32, 3>},
                                           {first_conv_kernel<false, 16, 0, true>, first_conv_kernel<false, 32, 0, true>, first_conv_kernel<false, 48, 0, true>,
                                            first_conv_kernel<false, 64, 0, true>, first_conv_kernel<false, 16, 1, true>, first_conv_kernel<false, 32, 3, true>}};
    static PerDeviceSmem configured[3][6];
    const int ki = first_variant(d, KP), si = stats ? 1 : pool ? 2 : 0;
    if (int rc = ensure_dynamic_smem(kernels[si][ki], 232448, configured[si][ki], "first_conv")) return rc;
    launch(kernels[si][ki], first_tc_grid(p.ntiles), ft_threads(stats != nullptr, KP, pool != nullptr), smem, st, p);
    count_launch();
    return check_launch("first_conv_kernel");
}

// dW / dB on the tensor cores need, on top of the forward's conditions, a power-of-two filter count (the producers'
// thread -> channel-chunk mapping) -- the same shapes conv_smallc.cu takes.
bool first_tc_bwd_eligible(const AetherConvDesc& d) {
    return first_tc_eligible(d) && smallc_conv_eligible(d) && d.Cout % 8 == 0;
}

// Workspace of the first-layer filter gradient: the per-CTA partials, then room for a bf16 copy of dy handed in by its
// producer ([P][ld], ld = Cout padded to 64) and for the column sums that come with it.
struct FirstDwLayout {
    size_t part_bytes, dy_off, colsum_off, total;
    int ld, rows_max;
};
static FirstDwLayout first_dw_layout(const AetherConvDesc& d, int K, long long P) {
    FirstDwLayout l;
    l.part_bytes = align_up((size_t)first_tc_grid((P + 127) / 128) * (K + 1) * d.Cout * sizeof(float), 1024);
    l.ld = (d.Cout + 63) / 64 * 64;
    l.dy_off = l.part_bytes;
    l.colsum_off = l.dy_off + align_up((size_t)P * l.ld * 2, 1024);
    l.rows_max = 8 * num_sms();
    l.total = l.colsum_off + align_up((size_t)l.rows_max * d.Cout * sizeof(float), 1024);
    return l;
}

size_t first_tc_bwd_workspace_bytes(const AetherConvDesc& d) {
    int K, KP, NT, Ho, Wo;
    if (!first_tc_bwd_eligible(d) || !first_tc_shape(d, K, KP, NT, Ho, Wo)) return 0;
    return first_dw_layout(d, K, 1LL * d.S * Ho * Wo).total;
}

bool first_tc_operand_layout(const AetherConvDesc& d, AetherOperandLayout* out) {
    int K, KP, NT, Ho, Wo;
    if (!first_tc_bwd_eligible(d) || !first_tc_shape(d, K, KP, NT, Ho, Wo)) return false;
    const FirstDwLayout l = first_dw_layout(d, K, 1LL * d.S * Ho * Wo);
    out->x_copy_offset = 0;
    out->x_copy_ld = 0;                     // the forward kernel gathers x itself: no copy of x to hand in
    out->dy_copy_offset = l.dy_off;
    out->dy_copy_ld = l.ld;
    out->dy_colsum_offset = l.colsum_off;
    out->dy_colsum_rows_max = l.rows_max;
    return true;
}

int first_tc_bwd_filter(const AetherConvDesc& d, const float* x, const float* dy, float* dw, float* db, void* ws,
                        size_t ws_bytes, int dy_colsum_rows, cudaStream_t st) {
    int K, KP, NT, Ho, Wo;
    if (!first_tc_bwd_eligible(d) || !first_tc_shape(d, K, KP, NT, Ho, Wo))
        return set_error(AE_UNSUPPORTED, "first_tc_bwd_filter: shape not supported");
    FirstDwParams p;
    memset(&p, 0, sizeof(p));
    p.g = first_geom(d, x, Ho, Wo);
    p.dy = dy; p.part = static_cast<float*>(ws); p.status = device_status_word();
    p.Cout = d.Cout; p.K = K; p.KP = KP;
    p.dblocks = (d.Cout + 127) / 128;
    p.P = 1LL * d.S * Ho * Wo;
    p.ntiles = (int)((p.P + 127) / 128);
    p.stage_bytes = FT_STAGE_BYTES * (1 + 2 * p.dblocks);
    const int tail = FD_TAIL;
    p.stages = (232448 - 1024 - tail) / p.stage_bytes;
    if (p.stages > 4) p.stages = 4;
    p.groups = p.stages < FD_MAX_GROUPS ? p.stages : FD_MAX_GROUPS;      // 1, 2 or 3: all divide FD_NP, FD_NP / groups is a multiple of 32
    const int grid = first_tc_grid(p.ntiles);
    const FirstDwLayout lay = first_dw_layout(d, K, p.P);
    const size_t need = dy_colsum_rows > 0 ? lay.total : (size_t)grid * (K + 1) * d.Cout * sizeof(float);
    if (!ws || ws_bytes < need) return set_error(AE_BAD_ARG, "conv workspace too small: %zu < %zu", ws_bytes, need);
    if (dy_colsum_rows > 0) {              // dy arrives as a bf16 copy with its column sums
        if (dy_colsum_rows > lay.rows_max)
            return set_error(AE_BAD_ARG, "aether_conv2d_bwd_ex: dy_colsum_rows %d outside [1, %d]", dy_colsum_rows, lay.rows_max);
        int rc0 = make_map_2d(&p.tm_dy, static_cast<uint8_t*>(ws) + lay.dy_off, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, lay.ld, p.P,
                              64, 128);
        if (rc0) return rc0;
        p.dy_bf16 = 1;
    }
    const int smem = 1024 + p.stages * p.stage_bytes + tail;
    using KernelFn = void (*)(const FirstDwParams);
    static const KernelFn kernels[6] = {first_dw_kernel<16, 0>, first_dw_kernel<32, 0>, first_dw_kernel<48, 0>,
                                        first_dw_kernel<64, 0>, first_dw_kernel<16, 1>, first_dw_kernel<32, 3>};
    static PerDeviceSmem configured[6];
    const int ki = first_variant(d, KP);
    if (int rc0 = ensure_dynamic_smem(kernels[ki], 232448, configured[ki], "first_dw")) return rc0;
    launch(kernels[ki], grid, FD_THREADS, smem, st, p);
    count_launch();
    int rc = check_launch("first_dw_kernel");
    if (rc) return rc;
    if (p.dy_bf16 && db)
        return smallc_reduce_partials(p.part, grid, K, d.Cout, dw, db, st,
                                      reinterpret_cast<const float*>(static_cast<uint8_t*>(ws) + lay.colsum_off), dy_colsum_rows);
    return smallc_reduce_partials(p.part, grid, K, d.Cout, dw, db, st);
}

}  // namespace aether
