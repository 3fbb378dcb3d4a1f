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
// half((residual + y) * norm_weight * 2^-(e + 3)) as the output and adds up every token's sum of squares.
// Consumer side (qkv, w13): the rows of the accumulator are scaled by 2^(e + 3) / rms before the output is rounded, which completes
// the normalisation of its input.
// 2^e <= rms < 2^(e + 1) of the row ahead of this addition (kLeastExponent at least), which both sides know.  What is stored has the
// size of a normalised row, an eighth of it, whatever the size of the rows and weights: it falls among fp16's subnormal numbers no sooner
// than what counts against the row's other values, and is finite as long as a value times its weight is below 2^19 * 2^e (a norm
// kernel's output is always; here a row of zeros may not become 2048 in one addition, nor one of rms 1 500000).

// A row's sum of squares.  Its parts (fp32 sums in a fixed order) are added as whole numbers, so that the order of the additions cannot
// change the result: each to `fine`, in units of 2^(2 e - 24), or, if it is 2^26 times 2^(2 e) or more, to `coarse`, in units of 2^-13.
// Either way it keeps the bits that count in an fp32 sum of the row.  Parts that are no numbers set the upper bit of `coarse`.
struct RowSquares {
    unsigned long long fine, coarse;  // of at most 2^12 parts (16384 values by four)
    int                exponent;      // e
    int                unused[3];     // 32 bytes: a sector
};
struct GemmNormFusion {
    __half*           residual    = nullptr;  // [T][N], producer
    const __half*     norm_weight = nullptr;  // [N], producer
    const RowSquares* ssq_before  = nullptr;  // [T] ahead of the addition, producer
    RowSquares*       ssq_out     = nullptr;  // [T], producer
    const RowSquares* ssq_in      = nullptr;  // [T], consumer
    float             inv_n       = 0.f;      // 1 / (length of the normalised row)
    float             eps         = 0.f;      // consumer
};
#ifdef __CUDACC__
constexpr int                kLeastExponent = -8, kMostExponent = 17;
constexpr unsigned long long kNotFinite     = 1ull << 63;
__device__ __forceinline__ float power_of_two(int e)  // in fp32's normal range
{
    return __int_as_float((e + 127) << 23);
}
__device__ __forceinline__ RowSquares load_row_squares(const RowSquares* at)
{
    RowSquares       r{};
    const ulonglong2 sums = __ldcg(reinterpret_cast<const ulonglong2*>(at));
    r.fine = sums.x, r.coarse = sums.y, r.exponent = __ldcg(&at->exponent);
    return r;
}
__device__ __forceinline__ float row_squares(const RowSquares& r)
{
    const float sum = __ull2float_rn(r.fine) * power_of_two(2 * r.exponent - 24);
    if (r.coarse == 0ull) return sum;
    return r.coarse >= kNotFinite ? __int_as_float(0x7fffffff) : sum + __ull2float_rn(r.coarse) * power_of_two(-13);
}
// floor(log2(rms)) from the mean square
__device__ __forceinline__ int row_exponent(float mean_square)
{
    return min(max((((__float_as_int(mean_square) >> 23) & 0xff) - 127) >> 1, kLeastExponent), kMostExponent);
}
// What a row is multiplied by: 2^(e + 3) / rms (consumer), 2^-(e + 3) (producer)
__device__ __forceinline__ float norm_row_scale(const GemmNormFusion& f, const RowSquares& r)
{
    return rsqrtf(row_squares(r) * f.inv_n + f.eps) * power_of_two(r.exponent + 3);
}
__device__ __forceinline__ float norm_row_down(const GemmNormFusion& f, const RowSquares& before)
{
    return power_of_two(-3 - row_exponent(row_squares(before) * f.inv_n));
}
__device__ __forceinline__ int exponent_of_down(float down)
{
    return 127 - 3 - (__float_as_int(down) >> 23);
}
// A part of a row's sum
__device__ __forceinline__ void add_row_squares(RowSquares* at, float part, float down)
{
    const float units = part * (down * down * power_of_two(30));
    if (units < power_of_two(50)) atomicAdd(&at->fine, __float2ull_rn(units));
    else if (part < power_of_two(60)) atomicAdd(&at->coarse, __float2ull_rn(part * power_of_two(13)));
    else atomicOr(&at->coarse, kNotFinite);
}
// The whole of it
__device__ __forceinline__ RowSquares whole_row_squares(float sum, float inv_n)
{
    RowSquares r{};
    r.exponent = row_exponent(sum * inv_n);
    if (sum < power_of_two(60)) r.fine = __float2ull_rn(sum * power_of_two(24 - 2 * r.exponent));
    else r.coarse = kNotFinite;
    return r;
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
