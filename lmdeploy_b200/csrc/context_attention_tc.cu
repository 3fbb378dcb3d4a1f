// Prefill (context) attention on the tcgen05 tensor core: causal softmax(q k^T / sqrt(d)) v over the KV cache read in
// place, fp16 or int8 cache, head size 128.  Same interface and results as context_attention.cu (the mma.sync kernel it
// replaces as the default); what it stands in for in the reference is described there
// (LlamaContextAttentionLayer<T>::fusedMultiHeadAttention, src/turbomind/models/llama/LlamaContextAttentionLayer.cc:257-313).
//
// One CTA = 128 queries of one (sequence, head); key / value tiles of 64 rows, double-buffered in shared memory in the
// 128-byte-swizzled layout the tensor core reads (two 64-wide blocks of the 128 head dimensions per tile).
//   warps 0-3   thread = query row = TMEM lane.  They copy the tiles (cp.async for fp16; int8 rows go through registers
//               and are dequantised on the way), and per tile: read the scores S from TMEM (tcgen05.ld), mask, online
//               softmax in the log2 domain with one thread per row (no shuffles), write the probabilities as fp16 into
//               TMEM (tcgen05.st) where the second product takes them as its A operand, and rescale the output
//               accumulator only when a row's running maximum moved by more than 2^8 (the accumulator is fp32).
//   warp 4      allocates TMEM (256 columns: S of two tiles, O 128; a tile's P takes its S's place); one lane issues S = Q K^T (both
//               operands from shared memory, M128 x N64 x K16, 8 per tile) and O += P V (A from TMEM, B = the value tile as an
//               MN-major operand, M128 x N128 x K16, 4 per tile) and commits to mbarriers.  The next tile's S is issued ahead of
//               this one's P V, so that it is computed under the softmax: with one S a tile's two products (576 and 280 cycles) and
//               its softmax came one after the other (fp16 cache, 8 x 2048 tokens, 32 heads 426 us, 373 so; 64 tokens behind 3000
//               68 and 57; int8, whose expansion by the same warps bounds it, 587 and 565).
// Two CTAs are resident per SM (97 KB of shared memory, 256 TMEM columns each), so one CTA's softmax overlaps the
// other's MMAs.  Tiles above the causal diagonal are never visited; the longest query tiles are scheduled first.
// Every barrier wait is bounded; on expiry a status bit is recorded and the CTA drains and leaves.
#include "common.cuh"
#include "context_attention.h"
#include "handle.h"
#include "tm_b200.h"

namespace tmb {
namespace {

constexpr int kD        = 128;
constexpr int kBM       = 128;  // queries per CTA
constexpr int kBN       = 64;   // keys per tile
constexpr int kRowThreads = 128;
constexpr int kThreads  = 160;
constexpr int kQBytes   = kBM * kD * 2;        // 32 KB: two blocks of [128 rows][128 B]
constexpr int kQBlock   = kBM * 128;           // 16 KB
constexpr int kTileBytes = kBN * kD * 2;       // 16 KB: two blocks of [64 rows][128 B]
constexpr int kTBlock   = kBN * 128;           // 8 KB
constexpr int kTmemCols = 256;
constexpr int kColS = 0, kColO = 128;  // two tiles' scores, whose place their probabilities take; the accumulator

struct Bars {
    uint64_t k_full[2];   // tile t's keys are in shared memory (128 arrivals)
    uint64_t s_full[2];   // S of tile t is in TMEM
    uint64_t p_full;      // P of tile t is in TMEM, its values in shared memory, O rescaled (128 arrivals)
    uint64_t pv_done;     // P V of tile t is in O
    uint64_t o_full;      // every product is done
    uint32_t tmem_base;
    int      dead;
};
constexpr int kSmemBytes = 1024 + kQBytes + 4 * kTileBytes + 128;

// byte offset of 16-byte chunk `chunk` (0..15 over the 128 head dimensions) of row `row`; `block_bytes` = rows x 128
__device__ __forceinline__ uint32_t sw_off(int row, int chunk, int block_bytes)
{
    return (uint32_t)((chunk >> 3) * block_bytes + row * 128 + (((chunk & 7) ^ (row & 7)) << 4));
}

__device__ __forceinline__ void cp_async16z(uint32_t dst, const void* src, int bytes)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// K-major operand (rows of 128 B, 8-row groups 1024 B apart), 128-byte swizzle
__device__ __forceinline__ uint64_t desc_kmajor(uint32_t addr)
{
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46)
           | ((uint64_t)2 << 61);
}
// MN-major operand: rows of the tile are K (keys), each row 128 B = 64 of the N (head dimension) values; groups of 8
// keys 1024 B apart, the second 64-wide block of N `block_bytes` further on
__device__ __forceinline__ uint64_t desc_mnmajor(uint32_t addr, uint32_t block_bytes)
{
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((block_bytes >> 4) & 0x3FFFu) << 16) | ((uint64_t)(1024 >> 4) << 32)
           | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

__device__ __forceinline__ void umma_ss(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc)
{
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
        "l"(da), "l"(db), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t acc)
{
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(tmem_d),
        "r"(tmem_a), "l"(db), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void umma_commit_to(uint64_t* bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void fence_async_smem()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_before()
{
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_after()
{
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// 32 consecutive 32-bit columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
          "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]),
        "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]),
        "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_wait_st()
{
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ float ex2(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint32_t pack2(float a, float b)
{
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// 4 int8 -> 4 halves, half(q * scale + zp) (llama_kernels.cu:309-316); the int -> float step through the mantissa of 2^23
__device__ __forceinline__ uint2 dequant4(uint32_t w, float scale, float zp)
{
    const uint32_t u  = w ^ 0x80808080u;
    const float    f0 = __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7540)) - 8388736.f;
    const float    f1 = __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7541)) - 8388736.f;
    const float    f2 = __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7542)) - 8388736.f;
    const float    f3 = __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7543)) - 8388736.f;
    uint2 r;
    r.x = pack2(__fmaf_rn(f0, scale, zp), __fmaf_rn(f1, scale, zp));
    r.y = pack2(__fmaf_rn(f2, scale, zp), __fmaf_rn(f3, scale, zp));
    return r;
}

template<bool INT8>
__global__ void __launch_bounds__(kThreads, 2) context_attention_tc_kernel(CtxParams p)
{
    extern __shared__ unsigned char smem_dyn[];
    pdl_wait();
    pdl_launch_dependents();
    const int tid = threadIdx.x, warp = tid >> 5;
    const int bi = blockIdx.z, h = blockIdx.y;
    const int qt    = gridDim.x - 1 - blockIdx.x;  // the longest (latest) query tiles first
    const int tok0  = p.cu_seqlens[bi];
    const int q_len = p.cu_seqlens[bi + 1] - tok0;
    const int ctx   = p.context_length[bi];
    const int hist  = ctx - q_len;
    const int q0    = qt * kBM;
    if (q0 >= q_len) return;  // the whole CTA, before anything is set up
    // keys any query of this tile may see; never past the rows a cache head holds
    const int kv_end  = min(min(ctx, p.max_seq_len), hist + min(q0 + kBM, q_len));
    const int n_tiles = (kv_end + kBN - 1) / kBN;
    const int kvh     = h / p.n_rep;

    const uint32_t raw  = smem_u32(smem_dyn);
    const uint32_t base = (raw + 1023u) & ~1023u;  // operand tiles on 1024-byte boundaries (the swizzle is a function of the address)
    unsigned char* sm   = smem_dyn + (base - raw);
    const uint32_t q_s  = base;
    const uint32_t kv_s = base + kQBytes;  // [buf][k | v]
    Bars*          bars = reinterpret_cast<Bars*>(sm + kQBytes + 4 * kTileBytes);

    if (tid == 0) {
        for (int i = 0; i < 2; ++i) mbar_init(&bars->k_full[i], kRowThreads), mbar_init(&bars->s_full[i], 1);
        mbar_init(&bars->p_full, kRowThreads);
        mbar_init(&bars->pv_done, 1);
        mbar_init(&bars->o_full, 1);
        bars->dead = 0;
        fence_mbar_init();
    }
    if (warp == 4) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)), "n"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_before();
    __syncthreads();
    tc_after();
    const uint32_t tmem = bars->tmem_base;

    if (warp < 4) {
        // ============================================================ copies, softmax, output: thread = query row
        const size_t         head_off = p.offset + (size_t)kvh * p.max_seq_len * kD;  // elements
        const unsigned char* k_base   = static_cast<const unsigned char*>(p.k_cache[bi]) + head_off * (INT8 ? 1 : 2);
        const unsigned char* v_base   = static_cast<const unsigned char*>(p.v_cache[bi]) + head_off * (INT8 ? 1 : 2);
        // tile t of the keys (which = 0) or the values (1) sits in buffer t & 1; tiles beyond the last one are not there
        auto load_f16 = [&](int t, int which) {
            const int key0 = t * kBN;
#pragma unroll
            for (int r = 0; t < n_tiles && r < 8; ++r) {
                const int    c = tid + r * kRowThreads, row = c >> 4, chunk = c & 15;
                const bool   ok  = key0 + row < kv_end;
                const size_t src = ((size_t)(ok ? key0 + row : 0) * kD + chunk * 8) * 2;
                cp_async16z(kv_s + (t & 1) * 2 * kTileBytes + which * kTileBytes + sw_off(row, chunk, kTBlock), (which ? v_base : k_base) + src,
                            ok ? 16 : 0);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        uint4 stage[2][4];  // int8 only: the next tiles on their way from global to shared memory
        auto  fetch_s8 = [&](int t, int which) {
            const int key0 = t * kBN;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int c = tid + r * kRowThreads, row = c >> 3, chunk = c & 7;
                stage[which][r] = make_uint4(0, 0, 0, 0);
                if (key0 + row < kv_end) stage[which][r] = *reinterpret_cast<const uint4*>((which ? v_base : k_base) + (size_t)(key0 + row) * kD + chunk * 16);
            }
        };
        auto store_s8 = [&](int t, int which) {
            const int      key0 = t * kBN;
            const float    scale = which ? p.v_scale : p.k_scale, zp = which ? p.v_zp : p.k_zp;
            unsigned char* dst = sm + kQBytes + (t & 1) * 2 * kTileBytes + which * kTileBytes;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int c = tid + r * kRowThreads, row = c >> 3, chunk = c & 7;
                uint4     lo = make_uint4(0, 0, 0, 0), hi = lo;
                if (key0 + row < kv_end) {  // rows past the end stay exact zeros (not the zero point)
                    const uint4 q = stage[which][r];
                    const uint2 a = dequant4(q.x, scale, zp), b = dequant4(q.y, scale, zp), c2 = dequant4(q.z, scale, zp), d = dequant4(q.w, scale, zp);
                    lo = make_uint4(a.x, a.y, b.x, b.y), hi = make_uint4(c2.x, c2.y, d.x, d.y);
                }
                *reinterpret_cast<uint4*>(dst + sw_off(row, 2 * chunk, kTBlock))     = lo;
                *reinterpret_cast<uint4*>(dst + sw_off(row, 2 * chunk + 1, kTBlock)) = hi;
            }
        };

        // ---- prologue: the query tile, two tiles of keys, one of values
        {
            const __half* qsrc = p.q + ((size_t)bi * p.H + h) * p.max_q_len * kD;
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                const int  c = tid + r * kRowThreads, row = c >> 4, chunk = c & 15;
                const bool ok = q0 + row < q_len;
                cp_async16z(q_s + sw_off(row, chunk, kQBlock), qsrc + (size_t)(ok ? q0 + row : 0) * kD + chunk * 8, ok ? 16 : 0);
            }
        }
        if (INT8) {
            fetch_s8(0, 0);
            fetch_s8(0, 1);
            store_s8(0, 0);
            asm volatile("cp.async.wait_all;" ::: "memory");
            fetch_s8(1, 0);
        }
        else {
            load_f16(0, 0);
            load_f16(1, 0);
            load_f16(0, 1);
            asm volatile("cp.async.wait_group 2;" ::: "memory");
        }
        fence_async_smem();  // copies and stores of this thread become visible to the tensor core's reads
        mbar_arrive(&bars->k_full[0]);

        const int      qi        = q0 + tid;
        const bool     row_live  = qi < q_len;
        const int      limit     = row_live ? min(hist + qi, kv_end - 1) : -1;  // last key this row may see
        const uint32_t lane_base = tmem + ((uint32_t)(warp * 32) << 16);
        float          m_used = -INFINITY, l = 0.f;
        bool           dead = false;
        for (int t = 0; t < n_tiles; ++t) {
            const int buf = t & 1;
            // int8 values are stored here already: the product on the tile before the last, which had their buffer, is complete
            if (INT8) store_s8(t, 1);
            if (t + 1 < n_tiles) {  // the next tile's scores are computed under this one's softmax
                if (INT8) store_s8(t + 1, 0);
                asm volatile("cp.async.wait_group 1;" ::: "memory");  // its keys have landed, this one's values may be on their way
                fence_async_smem();
                mbar_arrive(&bars->k_full[buf ^ 1]);
            }
            // the outcome is made uniform across the warp: the TMEM loads and stores below are warp-wide instructions
            if (!__all_sync(0xffffffffu, mbar_wait(&bars->s_full[buf], (t >> 1) & 1, p.max_wait_cycles))) {
                atomicOr(p.status, kStatusGemmPipeWait);
                *(volatile int*)&bars->dead = 1;
                dead = true;
                break;
            }
            tc_after();
            // S of this tile is complete: its keys' buffer is free
            if (INT8) {
                fetch_s8(t + 2, 0);
                fetch_s8(t + 1, 1);
            }
            else {
                load_f16(t + 2, 0);
            }
            const uint32_t scores = lane_base + kColS + buf * kBN;  // and, once they are read, the probabilities

            uint32_t s0[32], s1[32];
            tmem_ld32(scores, s0);
            tmem_ld32(scores + 32, s1);
            const int key0 = t * kBN;
            // raw scores stay as they are; the softmax scale goes into the exponent's multiply-add.  Only tiles that
            // touch the causal diagonal or the end of the keys mask anything (the same for every row of the CTA).
            float mx = -INFINITY;
            if (key0 + kBN - 1 > hist + q0 || key0 + kBN > kv_end || !row_live) {
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    if (key0 + i > limit) s0[i] = 0xff800000u;       // -inf
                    if (key0 + 32 + i > limit) s1[i] = 0xff800000u;
                }
            }
#pragma unroll
            for (int i = 0; i < 32; ++i) mx = fmaxf(mx, fmaxf(__uint_as_float(s0[i]), __uint_as_float(s1[i])));
            mx *= p.scale_log2;  // the scale is positive
            // the running maximum follows only when it is left behind by more than 2^8: p <= 256 fits fp16, the sums are
            // fp32, and the accumulator needs rescaling a few times per row instead of once per tile
            float alpha = 1.f;
            if (mx > m_used + 8.f) {
                alpha  = ex2(m_used - mx);  // 0 on the first tile
                m_used = mx;
            }
            const float nm  = m_used == -INFINITY ? 0.f : -m_used;
            float       sum = 0.f;
            uint32_t    pr[32];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const float a = ex2(fmaf(__uint_as_float(s0[2 * i]), p.scale_log2, nm)), b = ex2(fmaf(__uint_as_float(s0[2 * i + 1]), p.scale_log2, nm));
                const float c = ex2(fmaf(__uint_as_float(s1[2 * i]), p.scale_log2, nm)), d = ex2(fmaf(__uint_as_float(s1[2 * i + 1]), p.scale_log2, nm));
                sum += (a + b) + (c + d);
                pr[i]      = pack2(a, b);
                pr[16 + i] = pack2(c, d);
            }
            l = l * alpha + sum;
            // the accumulator and the buffer of the next values are free once the product on the tile before is complete
            if (t > 0 && !__all_sync(0xffffffffu, mbar_wait(&bars->pv_done, (t - 1) & 1, p.max_wait_cycles))) {
                atomicOr(p.status, kStatusGemmPipeWait);
                *(volatile int*)&bars->dead = 1;
                dead = true;
                break;
            }
            tc_after();
            if (t > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
#pragma unroll 1
                for (int c = 0; c < 4; ++c) {
                    uint32_t o[32];
                    tmem_ld32(lane_base + kColO + 32 * c, o);
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                    tmem_st32(lane_base + kColO + 32 * c, o);
                }
            }
            tmem_st32(scores, pr);
            asm volatile("cp.async.wait_group 1;" ::: "memory");  // this tile's values have landed, keys may be on their way
            fence_async_smem();
            tmem_wait_st();
            tc_before();
            mbar_arrive(&bars->p_full);
            if (!INT8) load_f16(t + 1, 1);
        }
        // ---- normalise and store: out[token, h * 128 + d]
        if (!dead && !__all_sync(0xffffffffu, mbar_wait(&bars->o_full, 0, p.max_wait_cycles))) {
            atomicOr(p.status, kStatusGemmTmemWait);
            dead = true;
        }
        tc_after();
        if (!dead && *(volatile int*)&bars->dead == 0) {
            const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
                uint32_t o[32];
                tmem_ld32(lane_base + kColO + 32 * c, o);
                if (row_live) {
                    __half* dst = p.out + ((size_t)(tok0 + qi) * p.H + h) * kD + 32 * c;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        uint4 v;
                        v.x = pack2(__uint_as_float(o[8 * i]) * inv, __uint_as_float(o[8 * i + 1]) * inv);
                        v.y = pack2(__uint_as_float(o[8 * i + 2]) * inv, __uint_as_float(o[8 * i + 3]) * inv);
                        v.z = pack2(__uint_as_float(o[8 * i + 4]) * inv, __uint_as_float(o[8 * i + 5]) * inv);
                        v.w = pack2(__uint_as_float(o[8 * i + 6]) * inv, __uint_as_float(o[8 * i + 7]) * inv);
                        *reinterpret_cast<uint4*>(dst + 8 * i) = v;
                    }
                }
            }
        }
    }
    else {
        // ============================================================ MMA issuer: one elected lane of the warp runs the whole loop, as a vote
        // between its steps would stand in a chain that nothing hides where an SM has one CTA
        if (elect_one()) {
            const uint32_t idesc_qk = (1u << 4) | ((uint32_t)(kBN >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
            const uint32_t idesc_pv = (1u << 4) | (1u << 16) | ((uint32_t)(kD >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);  // B is MN-major
            auto           issue_scores = [&](int t) {
                const int buf = t & 1;
                if (!mbar_wait(&bars->k_full[buf], (t >> 1) & 1, p.max_wait_cycles)) return false;
                tc_after();
#pragma unroll
                for (int blk = 0; blk < 2; ++blk) {
                    const uint64_t dq = desc_kmajor(q_s + blk * kQBlock), dk = desc_kmajor(kv_s + buf * 2 * kTileBytes + blk * kTBlock);
#pragma unroll
                    for (int j = 0; j < 4; ++j) umma_ss(tmem + kColS + buf * kBN, dq + (uint64_t)(2 * j), dk + (uint64_t)(2 * j), idesc_qk, (blk | j) ? 1u : 0u);
                }
                umma_commit_to(&bars->s_full[buf]);
                return true;
            };
            bool ok = issue_scores(0);
            for (int t = 0; t < n_tiles && ok; ++t) {
                // The columns that tile t + 1's scores take hold tile t - 1's probabilities: not before their product is complete (products
                // of different shapes and accumulators are not promised to run in order)
                if (t > 0 && t + 1 < n_tiles) ok = mbar_wait(&bars->pv_done, (t - 1) & 1, p.max_wait_cycles);
                ok = ok && (t + 1 >= n_tiles || issue_scores(t + 1)) && mbar_wait(&bars->p_full, t & 1, p.max_wait_cycles);
                if (!ok) break;
                tc_after();
                const uint64_t dv = desc_mnmajor(kv_s + (t & 1) * 2 * kTileBytes + kTileBytes, kTBlock);
#pragma unroll
                for (int j = 0; j < 4; ++j) umma_ts(tmem + kColO, tmem + kColS + (t & 1) * kBN + 8 * j, dv + (uint64_t)(128 * j), idesc_pv, (t | j) ? 1u : 0u);
                umma_commit_to(&bars->pv_done);
            }
            if (!ok) {
                atomicOr(p.status, kStatusGemmPipeWait);
                *(volatile int*)&bars->dead = 1;
            }
            umma_commit_to(&bars->o_full);  // arrives when everything issued so far is complete (also on the give-up path)
        }
        __syncwarp();
    }

    tc_before();
    __syncthreads();
    if (warp == 4) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(kTmemCols) : "memory");
    }
}

}  // namespace

cudaError_t context_attention_tc_launch(const CtxParams& p, bool int8, int batch, cudaStream_t st)
{
    auto kernel = int8 ? context_attention_tc_kernel<true> : context_attention_tc_kernel<false>;
    // per call, like every attribute in this library that depends on the current device; cheap next to the kernel
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e != cudaSuccess) return e;
    const dim3 grid((p.max_q_len + kBM - 1) / kBM, p.H, batch);
    return launch_kernel(kernel, grid, dim3(kThreads), kSmemBytes, st, g_pdl != 0, p);
}

}  // namespace tmb
