// W4A16 GEMM for many tokens: the packed weight is expanded once, to fp16 rows in scratch, and multiplied by the dense
// kernel's pairs of CTAs (gemm_dense.cu).  The kernel that expands while it multiplies (gemm_s4_f16_tc.cu) does so again for
// every 128 tokens: from some hundreds of tokens on the expansion, not the tensor core, is what its time goes to.
// The numbers are the same: fp16((q - z) * s) on fp16 activations, fp32 sums.
#include "common.cuh"
#include "gemm_dense.h"
#include "gemm_s4_f16.h"
#include "handle.h"
#include "tm_b200.h"

#include <algorithm>

namespace tmb {
namespace {

constexpr int kTileBytes = 512;  // 32 output features x 32 k
constexpr int kWarps     = 8;

__device__ __forceinline__ uint32_t scaled(uint32_t x, uint32_t s)
{
    uint32_t r;
    asm("mul.ftz.f16x2 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(s));
    return r;
}

// Bound by the writes (2 bytes per weight, 0.5 read): 0.51 us per million weights, 4.9 TB/s.  A warp expands 32 features x one 128-row group: the fragments of a slab
// are pieces of 4 bytes (two k) of a feature, piece (k16, half, c) in lane c of the four that share the feature; the four
// lanes trade pieces so that each holds 16 consecutive bytes, and a store covers whole 64-byte runs.
__global__ void __launch_bounds__(kWarps * 32) expand_s4_kernel(__half* w, const unsigned char* packed, const __half2* zs, int n_tiles, int N, int K, int tile0,
                                                              int tiles)
{
    pdl_wait();  // the rows of the product before lie in the same scratch
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, c = lane & 3;
    const int i = blockIdx.x * kWarps + warp, groups = K / 128;
    if (i >= tiles * groups) return;
    const int g = i / tiles, tile = tile0 + i % tiles;
    uint4     in[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        in[s] = __ldcs(reinterpret_cast<const uint4*>(packed + ((size_t)(4 * g + s) * n_tiles + tile) * kTileBytes) + lane);
    }
    const __half2* q = zs + (size_t)g * N + tile * 32;
    uint32_t       z1024[2], nz64[2], s_lo[2], s_hi[2];
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        const __half2 lo = q[a * 16 + r], hi = q[a * 16 + r + 8];
        const __half2 zl = __half2half2(__hadd(__low2half(lo), __float2half_rn(960.f))), zh = __half2half2(__hneg(__low2half(hi)));
        const __half2 sl = __half2half2(__high2half(lo)), sh = __half2half2(__high2half(hi));
        z1024[a] = reinterpret_cast<const uint32_t&>(zl), nz64[a] = reinterpret_cast<const uint32_t&>(zh);
        s_lo[a] = reinterpret_cast<const uint32_t&>(sl), s_hi[a] = reinterpret_cast<const uint32_t&>(sh);
    }
    // pieces x[j] of lane c belong to place 4 j + c -> lane c gets places 4 c .. 4 c + 3
    auto trade = [&](uint32_t (&x)[4]) {
        const bool odd = c & 1, up = c & 2;
        uint32_t   t0 = odd ? x[0] : x[1], t1 = odd ? x[2] : x[3];
        t0 = __shfl_xor_sync(0xffffffffu, t0, 1), t1 = __shfl_xor_sync(0xffffffffu, t1, 1);
        if (odd) {
            x[0] = t0, x[2] = t1;
        }
        else {
            x[1] = t0, x[3] = t1;
        }
        uint32_t u0 = up ? x[0] : x[2], u1 = up ? x[1] : x[3];
        u0 = __shfl_xor_sync(0xffffffffu, u0, 2), u1 = __shfl_xor_sync(0xffffffffu, u1, 2);
        if (up) {
            x[0] = u0, x[1] = u1;
        }
        else {
            x[2] = u0, x[3] = u1;
        }
    };
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const uint32_t wv[4] = {in[s].x, in[s].y, in[s].z, in[s].w};
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            uint32_t f0[4], f1[4];
            unpack_s4_minus_zero(wv[a], z1024[a], nz64[a], f0);      // k 0..15 of the slab
            unpack_s4_minus_zero(wv[2 + a], z1024[a], nz64[a], f1);  // k 16..31
            uint32_t lo[4] = {scaled(f0[0], s_lo[a]), scaled(f0[2], s_lo[a]), scaled(f1[0], s_lo[a]), scaled(f1[2], s_lo[a])};
            uint32_t hi[4] = {scaled(f0[1], s_hi[a]), scaled(f0[3], s_hi[a]), scaled(f1[1], s_hi[a]), scaled(f1[3], s_hi[a])};
            trade(lo);
            trade(hi);
            __half* dst = w + (size_t)((tile - tile0) * 32 + a * 16 + r) * K + g * 128 + s * 32 + c * 8;
            *reinterpret_cast<uint4*>(dst)                 = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            *reinterpret_cast<uint4*>(dst + (size_t)8 * K) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        }
    }
}

}  // namespace

// Which way is faster, by models of both in microseconds: the plan's of expanding while multiplying; expanding first, 2.5 bytes
// per weight beside the dense product.  The line lies between 2000 and 4000 tokens on most shapes.  Both sides, us, expanding first and
// while multiplying: 22016 x 4096 with 1536 / 2048 / 8192 / 16384 tokens 254 / 337 / 1216 / 2524 and 233 / 331 / 1318 / 2626;
// 8192 x 28672 with 1024 / 2048 tokens 515 / 912 and 420 / 789; 57344 x 8192 with 8192 / 16384 tokens 7005 / 14353 and 7792 / 15555.
int gemm_expanded_columns(const tm_handle* h, int N, int T, int K)
{
    if (T <= 128 || K % 128 || N % 32 || h->sm_count < 2) return 0;
    const int room = (int)std::min<size_t>(h->scratch_bytes / ((size_t)K * 2) / 256 * 256, 1u << 30);
    if (room < 256) return 0;
    const int pieces  = (N + room - 1) / room;
    const int columns = std::min(room, ((N + pieces - 1) / pieces + 255) / 256 * 256);
    double first = -36.7;
    for (int n0 = 0; n0 < N; n0 += columns) {
        const int n = std::min(columns, N - n0);
        first += 48.2 + 0.42e-6 * n * K + 0.98 * dense_pair_us(T, n, (K + 63) / 64, h->sm_count);
    }
    const double along = gemm_tc_plan(N, T, K, h->sm_count, true).us;
    return first < along ? columns : 0;
}

int gemm_expanded_launch(tm_handle* h, const GemmTcParams& p, int columns, cudaStream_t st, bool pdl)
{
    __half* const w = static_cast<__half*>(h->scratch);
    for (int n0 = 0; n0 < p.N; n0 += columns) {
        const int n = std::min(columns, p.N - n0), units = n / 32 * (p.K / 128);
        const cudaError_t e = launch_kernel(expand_s4_kernel, dim3((units + kWarps - 1) / kWarps), dim3(kWarps * 32), 0, st, pdl, w, p.A,
                                            reinterpret_cast<const __half2*>(p.Q), p.N / 32, p.N, p.K, n0 / 32, n / 32);
        if (e != cudaSuccess) {
            h->last_cuda_error = (int)e;
            return TM_ERR_CUDA;
        }
        ++h->launches;
        DenseGemm g;
        g.w = w, g.x = p.X, g.ldw = p.K, g.ldx = p.K, g.tokens = p.T, g.n_out = n, g.k = p.K;
        if (p.fused_silu) {
            g.ep.kind = DenseKind::kInput, g.ep.split = 0, g.ep.act = p.C + n0 / 2, g.ep.act_ld = p.N / 2, g.ep.activation = DenseActivation::kSiluHalf;
        }
        else {
            g.ep.kind = DenseKind::kStore, g.ep.out = p.C + n0, g.ep.out_ld = p.N;
        }
        const int rc = dense_gemm_f16(h, g, st, pdl);
        if (rc != TM_OK) return rc;
    }
    return TM_OK;
}

}  // namespace tmb
