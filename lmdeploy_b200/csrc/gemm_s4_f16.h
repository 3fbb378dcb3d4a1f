// Internal interface between the C ABI (api.cu) and the W4A16 GEMM kernels.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

struct tm_handle;

namespace tmb {

// Residual add + RMSNorm folded into the GEMMs on either side in the decode step (decode driver only).
// Producer side (o_proj, w2): whoever has the whole sum of an output adds the residual, stores it, writes
// half((residual + y) * norm_weight) as the output and adds up every token's sum of squares in 2^-20 fixed point
// (integer atomics: the order of the additions cannot change the result).
// Consumer side (qkv, w13): the rows of the accumulator are scaled by rsqrt(ssq[t] * 2^-20 * inv_n + eps) before the
// output is rounded, which completes the normalisation of its input.
struct GemmNormFusion {
    __half*                   residual    = nullptr;  // [T][N], producer
    const __half*             norm_weight = nullptr;  // [N], producer
    unsigned long long*       ssq_out     = nullptr;  // [T], producer
    const unsigned long long* ssq_in      = nullptr;  // [T], consumer
    float                     inv_n       = 0.f;      // 1 / (length of the normalised row), consumer
    float                     eps         = 0.f;
};
#ifdef __CUDACC__
// consumer: 1 / rms of row t
__device__ __forceinline__ float norm_row_scale(const GemmNormFusion& f, int t)
{
    return rsqrtf((float)__ldcg(f.ssq_in + t) * (1.f / 1048576.f) * f.inv_n + f.eps);
}
#endif

// ---- small-token (HBM-bound) kernel -----------------------------------------------------
struct GemmSmallParams {
    __half*              C;
    const unsigned char* A;  // runtime int4 layout, [K/32][N/32][512 B]
    const unsigned char* X;  // half [T, K]
    const unsigned char* Q;  // half2 [K/128, N]
    float*               workspace;
    int*                 counters;
    unsigned*            status;
    int                  N, T, K;
    int                  fused_silu;
    // filled in by gemm_small_launch from the plan
    int units_per_cta, total_units, slots_per_chunk, n_col_tiles, stages, cluster;
    int late_weight;  // 1: the kernel ahead may write the weight (a dependent launch waits before it reads any)
    GemmNormFusion norm;  // all null: a plain GEMM
};

struct GemmSmallPlan {
    int    nt;             // 8-token MMA tiles per pass (1, 2 or 4)
    int    t_chunks;       // passes over the weight (grid.y)
    int    n_col_tiles;    // 512-column tiles
    int    total_units;    // 64x512 weight units
    int    units_per_cta;
    int    ctas;
    int    slots_per_chunk;  // split-K scratch slots per token chunk (= ctas + n_col_tiles)
    int    stages;
    int    cols_tiles;     // 1 or 2: the column-owner kernel runs instead, on strips of that many 32-column tiles (up to 16 tokens
                           // with one, 8 with two); 0: the split-K kernel
    int    cols_cluster;   // CTAs that share a strip, all strips' at once on the device (or 1)
    size_t smem_bytes;
    size_t workspace_floats;
    size_t counter_ints;
};

size_t        gemm_small_smem_bytes(int nt);
GemmSmallPlan gemm_small_plan(int N, int T, int K, int sm_count, int max_smem, int cols_variant = 1);
cudaError_t   gemm_small_prepare(int max_smem);
cudaError_t   gemm_small_launch(const GemmSmallPlan& plan, GemmSmallParams p, cudaStream_t st, bool pdl = false);

// ---- tensor-core (tcgen05) kernel for more than 16 tokens ---------------------------------
struct GemmTcParams {
    __half*              C;
    const unsigned char* A;
    const unsigned char* X;
    const unsigned char* Q;
    float*               workspace;
    int*                 counters;
    unsigned*            status;
    int                  N, T, K;
    int                  fused_silu;
    // filled in by gemm_tc_launch from the plan
    int units_per_cta, total_units, slots_per_chunk, n_col_tiles, token_tile, parts_per_tile;
    int       late_weight;      // 1: the kernel ahead may write the weight (a dependent launch waits before it reads any)
    int       last_sums;        // 1: a split tile is reduced by the CTA that is done last, without a wait (GemmNormFusion: its consumer only)
    long long max_wait_cycles;  // bound of the wait for the partners of a split tile; 0 = the default
    GemmNormFusion norm;        // all null: a plain GEMM
};

struct GemmTcPlan {
    int    token_tile;     // UMMA N: tokens per pass, multiple of 16, <= 128
    int    t_chunks;       // passes over the weight (grid.y), 128 tokens each
    int    n_col_tiles;    // 256-feature tiles
    int    total_units;    // 128x256 weight units
    int    units_per_cta;
    int    parts_per_tile;  // CTAs per column tile (each with up to units_per_cta groups of it); 0 = the flat unit list cut evenly
    int    ctas;
    int    slots_per_chunk;
    int    last_sums;      // see GemmTcParams
    size_t smem_bytes;
    size_t workspace_floats;
    size_t counter_ints;
    double us;             // the launch's time by the plan's model
};

size_t      gemm_tc_smem_bytes(int token_tile);
// `balance` = false: never cuts tiles where there are at least as many as SMs (what tm_gemm_s4_f16_workspace_bytes counts on)
GemmTcPlan  gemm_tc_plan(int N, int T, int K, int sm_count, bool balance);
// true when every output tile of the plan is reduced by reduce_share (the only place that applies GemmNormFusion)
bool        gemm_tc_all_tiles_split(const GemmTcPlan& plan, int K);
cudaError_t gemm_tc_prepare(int max_smem);
cudaError_t gemm_tc_launch(const GemmTcPlan& plan, GemmTcParams p, cudaStream_t st, bool pdl = false);

// ---- many tokens: the weight expanded to fp16 rows in the handle's scratch, then a dense product (gemm_s4_f16_expand.cu) ----
// output columns that are expanded and multiplied at a time (all, or pieces that fit the scratch); 0: the other kernel is faster
int gemm_expanded_columns(const tm_handle* h, int N, int T, int K);
// C, A, X, Q, N, T, K and fused_silu of `p` are read
int gemm_expanded_launch(tm_handle* h, const GemmTcParams& p, int columns, cudaStream_t st, bool pdl);

}  // namespace tmb
