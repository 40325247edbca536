// Host-side helpers shared by the tensor-core convolution files.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <string.h>

#include "common.cuh"

namespace aether {

// One M tile is a box of BN images x BH rows x BW columns of output pixels.
struct PixelTiling {
    int BW, BH, BN, rows;
    int tiles_w, tiles_h, tiles_n;
    long long total() const { return 1LL * tiles_w * tiles_h * tiles_n; }
};

// The plan of a shape: working one out costs some ten microseconds of host time, as much as the launches of a small layer,
// and a network asks for the same few shapes again on every pass (workspace size, operand layout, statistics blocks, forward,
// backward): each host thread keeps the plans it used last, direct-mapped.  A plan depends on the shape and the device only.
template <typename Plan, Plan (*COMPUTE)(const AetherConvDesc&)>
const Plan& cached_plan(const AetherConvDesc& d) {
    struct Slot {
        AetherConvDesc key;
        int dev = -1;
        Plan plan;
    };
    static thread_local Slot slots[64];
    const int dev = current_device();
    uint32_t h = 2166136261u;
    const int32_t* f = reinterpret_cast<const int32_t*>(&d);
    for (size_t i = 0; i < sizeof(d) / sizeof(int32_t); ++i) h = (h ^ (uint32_t)f[i]) * 16777619u;
    Slot& s = slots[(h ^ (h >> 16)) & 63u];
    if (s.dev != dev || memcmp(&s.key, &d, sizeof(d)) != 0) {
        s.plan = COMPUTE(d);
        s.key = d;
        s.dev = dev;
    }
    return s.plan;
}

int num_sms();
// Whether this device can co-schedule the CTA pairs (clusters of two CTAs with ~210 KB of shared memory each) the
// cta_group::2 kernels are launched as, on every pair of SMs; looked up once per device.  False keeps the single-CTA forms.
bool cta_pairs_available();
// NHWC tensor seen as 4-D (C, W, H, N), box (box_c, BW, BH, BN); 128-byte swizzle unless told otherwise.
int make_map_nhwc(CUtensorMap* m, const void* base, CUtensorMapDataType dt, int elt, int C, int W, int H, int N,
                  int box_c, int BW, int BH, int BN, CUtensorMapSwizzle swz = CU_TENSOR_MAP_SWIZZLE_128B);
// Tensor map of any rank: sizes, byte strides of all dimensions but the innermost, box and element strides.
int make_map(CUtensorMap* m, const void* base, CUtensorMapDataType dt, int rank, const cuuint64_t* dims, const cuuint64_t* strides,
             const cuuint32_t* box, const cuuint32_t* estr, CUtensorMapSwizzle swz);
// Row-major matrix (inner = K elements contiguous, `rows` rows), box (box_k, box_rows); 128-byte swizzle unless told otherwise.
int make_map_2d(CUtensorMap* m, const void* base, CUtensorMapDataType dt, int elt, int inner, long long rows, int box_k,
                int box_rows, CUtensorMapSwizzle swz = CU_TENSOR_MAP_SWIZZLE_128B);
// What the per-tap kernel (conv_tc.cu) takes for a product, in clocks: padded columns, tiles of 128 pixels, 128-byte chunks of K over all taps.
double per_tap_clocks(int n_padded, long long m_tiles, int kiters);
// Halo-reuse kernel (conv_halo.cu): launches and sets *used when the problem fits it, else leaves *used false.  tap_n, tap_tiles: the per-tap kernel's
// padded columns and tiles of pixels.
int run_halo_igemm(bool tf32, const void* in, int in_C, int in_H, int in_W, int S, const void* wmat, int w_inner,
                   int rows_per_tap, int taps, float* out, int out_C, int out_H, int out_W, int n_padded, int tap_n, long long tap_tiles, int fH, int fW,
                   int padT, int padL, int flip, int k_real, const float* bias, float* stats, int prof_kind, cudaStream_t st,
                   bool* used);
// Partial-statistics blocks ([block][3][out_C]: count, mean, M2) the halo kernel writes when `stats` is given; 0 when
// the halo kernel does not take the problem.
long long halo_igemm_stats_blocks(bool tf32, int in_C, int S, int taps, int out_C, int out_H, int out_W, int n_padded,
                                  int tap_n, long long tap_tiles, int fH, int fW);
// What the halo kernel takes for such a problem, in clocks; 0 when it does not take it.
double halo_igemm_clocks(bool tf32, int in_C, int S, int taps, int out_C, int out_H, int out_W, int n_padded, int tap_n, long long tap_tiles, int fH, int fW);

// Halo-reuse dW kernel (conv_halo_dw.cu), bf16 shadows with 64-channel blocks.  `part` must have room for
// max_splits split slices; the split count actually used is returned in *splits_out.
int run_halo_dw(const void* x_sh, int Cin_p, int H, int W, int S, const void* dy_sh, int Cout_p, int Ho, int Wo, int fH,
                int fW, int padH, int padW, float* part, int max_splits, int* splits_out, cudaStream_t st, bool* used);

// conv_dw_rows.cu: dW with dy as the M operand and the taps of a filter row as N (3-row filters, bf16).
int rows_dw_max_splits(int Cin_p, int Cout_p, int Ho, int Wo, int S, int fH, int fW);
int run_rows_dw(const void* x_sh, int Cin_p, int H, int W, int S, const void* dy_sh, int Cout_p, int Ho, int Wo, int fH,
                int fW, int padH, int padW, float* part, int* splits_a, int* splits_b, int* tap_split, cudaStream_t st,
                bool* used);

// dw[tap][c][d] = sum over splits of part[split][tap * cblocks + c / UC][c % UC][d] (rows of `ldn`, a multiple of 4) and, when
// asked for, db from `db_rows` rows of column sums (conv_tc.cu).
int dw_reduce(const float* part, float* dw, int splits, int U, int UC, int ldn, int cblocks, int taps, int Cin, int Cout, int tap_split,
              int splits2, const float* dbpart, int db_rows, float* db, cudaStream_t st);

// Rows of a strip for the dW kernels that walk images in strips: among the heights that leave three stages in `avail` bytes (two, if there are
// none) the one with the fewest steps of 16 pixels over an image, two more per strip for what a strip costs by itself.  stage(bh): bytes of a stage.  (The
// highest strip instead: 16 rows in strips of 12 are a third padding; dW of 4238 x 16x16 64->64 190 us, in strips of 8 113.)
template <typename Stage>
static inline int pick_strip_rows(int Ho, int Wp, int avail, Stage stage, int* stages) {
    int best = 0;
    for (int most = 3; most >= 2 && best == 0; --most) {
        long long best_cost = 0;
        for (int bh = Ho < 16 ? Ho : 16; bh >= 1; --bh) {
            const int stg = avail / stage(bh);
            const long long cost = 1LL * ceil_div(Ho, bh) * (ceil_div(bh * Wp, 16) + 2);
            if (stg < most || (best != 0 && cost >= best_cost)) continue;
            best = bh;
            best_cost = cost;
            *stages = stg > 4 ? 4 : stg;
        }
    }
    return best;
}

// MMAs (32 bytes of K each) that the last of `kchunks` 128-byte chunks needs when only k_real of the channels are not padding.
static inline int last_ksteps(int k_real, int kchunks, int KC) {
    const int rest = k_real - (kchunks - 1) * KC, step = KC / 4;
    return rest >= KC ? 4 : rest <= step ? 1 : (rest + step - 1) / step;
}

}  // namespace aether
