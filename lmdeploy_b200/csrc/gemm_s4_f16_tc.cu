// W4A16 GEMM from 9 to 17 tokens on (api.cu): tcgen05 tensor-core tiles with the accumulators in TMEM.
//
// A CTA computes C^T tiles of 256 output features (two 128-feature UMMA tiles that share one
// activation slice) x up to 128 tokens.  Work units are (256-feature tile, 128-row quantisation
// group); a CTA has a whole tile, or the units of all tiles are cut evenly (gemm_tc_plan).  Warp roles:
//   warp 0       an elected lane streams the activation slices: one tensor-map copy (TMA, 128-byte
//                swizzle, tokens beyond T read as zero) per unit, completion on an mbarrier
//   warps 1, 2   one issuer per 128-feature tile (warp 1 also allocates TMEM): an elected lane issues
//                tcgen05.mma (M = 128, N = token tile, K = 16 per instruction, fp16 x fp16 -> fp32, A
//                from TMEM, B from shared memory) and commits completions to mbarriers
//   warps 3..18  two teams of eight, one per 128-feature tile; four warps of a team (32 features each)
//                take the even units, four the odd ones.  A warp takes its words from shared memory and expands them: lop3 nibble
//                unpack, exact (q - z) in fp16, one fp16 multiply by the scale (bit-identical to the
//                reference's dequantised weight, kernels/gemm_s_f16/common.h:115-156, 218-235),
//                tcgen05.st of the fragments straight into TMEM, from where the tensor core takes
//                its A operand (no shared-memory round trip); at the end of a column tile the
//                warps read the accumulators with tcgen05.ld and store C (optionally through the
//                SiLU(gate) * up epilogue) or the split-K partial
//   warp 19      an elected lane streams the packed weight: a box of the weight and one of {zero, scale} per unit
// What bounds it.  With few tokens the bytes of a unit take 0.4 us, its expansion 0.5-0.55 (65 % of the issue slots; 375 warp
// instructions per warp and unit, of which 208 unpack and scale).  Copies by the expanding warps (cp.async, 64-bit addresses) and
// issuers that voted between the steps of a unit cost 82 more instructions and left the issuing lane, a chain of 1100 cycles a unit,
// as the bound.  57344 x 8192, 16 / 64 tokens: 85 / 93 -> 67 / 76 us in a row of dependent launches over weights beyond the L2 (3.7 TB/s).
// Partial tiles of CTAs that share a column tile meet in scratch memory; every CTA of the tile then
// sums its own share of the feature rows in a fixed order.  Every wait is bounded.
//
// Replaces the large-n end of GemmS4F16::Run (src/turbomind/kernels/gemm_s_f16/gemm_s4_f16.cu:
// 208-234; mma.sync tiles of gemm_template.h:338-444).
#include "common.cuh"
#include "handle.h"
#include "gemm_s4_f16.h"

#include <algorithm>
#include <array>
#include <cuda.h>  // CUtensorMap (types only: the encoder is looked up through the runtime)

namespace tmb {
namespace {

template<int V>
struct Int {
    static constexpr int value = V;
};
constexpr int kTileN     = 128;  // output features per UMMA tile (UMMA M)
constexpr int kTeams     = 2;    // UMMA tiles per CTA tile
constexpr int kSuperN    = kTileN * kTeams;
constexpr int kGroup     = 128;  // K extent of a unit
constexpr int kTileBytes = 512;
constexpr int kSlabs     = kGroup / 32;
constexpr int kSlabBytes = kSuperN / 32 * kTileBytes;  // the packed weight of a 32-row slab of a unit: eight tiles, contiguous
constexpr int kWStage    = kSlabs * kSlabBytes + kSuperN * 4;  // a unit's packed weight and its row of {zero, scale}
constexpr int kWST       = 6;                    // stages of packed weight: 104 KB on their way, 44 KB hide the memory's latency
// Tokens of a tile decide how TMEM is shared out: two accumulators, and stages of expanded weight in the rest
template<bool kWide>
struct Shape {
    static constexpr int kAcc   = kWide ? 128 : 64;   // TMEM columns of an accumulator: the largest token tile
    // From 65 tokens on the products of a unit take as long as its expansion; stages of half a unit let the two overlap where there
    // is no room for a third whole one (4096 x 4096, 735 tokens: 39 us with two whole ones, 34 with four halves).
    static constexpr int kStageK = kWide ? 64 : 128;  // k values of a stage
    static constexpr int kParts  = kGroup / kStageK;  // stages of a unit
    static constexpr int kACols  = kStageK / 2;       // TMEM columns of a stage (fp16 pairs)
    static constexpr int kAST    = kWide ? 4 : 3;     // stages per team
    static constexpr int kXST    = kWide ? 3 : 6;     // activation stages in shared memory
};
constexpr int kASTMax = 4, kXSTMax = 6;
constexpr int kTeamWarps = 8;
constexpr int kDqWarps   = kTeams * kTeamWarps;
constexpr int kDqThreads = kDqWarps * 32;
constexpr int kIssuers   = kTeams;
constexpr int kDqWarp0   = 1 + kIssuers;         // first expanding warp
constexpr int kWLoadWarp = kDqWarp0 + kDqWarps;  // loader of the packed weight
constexpr int kThreads   = (kWLoadWarp + 1) * 32;
constexpr int kTmemCols  = 512;                  // accumulators + expanded-weight stages, power of two

struct Bars {
    uint64_t a_full[kTeams][kASTMax], a_empty[kTeams][kASTMax];
    uint64_t x_full[kXSTMax], x_empty[kXSTMax];
    uint64_t w_full[kWST], w_empty[kWST];
    uint64_t acc_full[kTeams], acc_empty[kTeams];  // per team
    uint32_t tmem_base;
    int      flag;
    float    row_scale[128];  // factor of a token (either side of a folded norm)
};
constexpr int kSquaresLd = 33;  // sums of squares of a token (producer of a folded norm): a share of a split tile has at most 32 quads of features

__device__ __forceinline__ uint64_t make_desc(uint32_t smem_addr)
{
    // K-major, 128-byte swizzle: 8-row groups 1024 B apart (SBO), leading offset 1, descriptor version 1
    return (uint64_t)((smem_addr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46)
           | ((uint64_t)2 << 61);
}

// Four MMAs: one 64-wide K block (four 16-wide steps) of a unit, operands precomputed so that an MMA costs the
// issuing thread three instructions.  `first`: the first MMA overwrites the accumulator.
__device__ __forceinline__ void umma_f16_ts_x4(uint32_t tmem_d, uint32_t tmem_a, uint32_t desc_lo, uint32_t desc_hi, uint32_t idesc,
                                               uint32_t first)
{
    asm volatile(
        "{\n"
        ".reg .pred p, t;\n"
        ".reg .b64 d;\n"
        ".reg .b32 a, l;\n"
        "setp.eq.b32 p, %5, 0;\n"      // accumulate unless first
        "setp.eq.b32 t, 0, 0;\n"       // always accumulate
        "mov.b64 d, {%2, %3};\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], d, %4, p;\n"
        "add.u32 a, %1, 8;\n  add.u32 l, %2, 2;\n  mov.b64 d, {l, %3};\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [a], d, %4, t;\n"
        "add.u32 a, %1, 16;\n add.u32 l, %2, 4;\n  mov.b64 d, {l, %3};\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [a], d, %4, t;\n"
        "add.u32 a, %1, 24;\n add.u32 l, %2, 6;\n  mov.b64 d, {l, %3};\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [a], d, %4, t;\n"
        "}\n" ::"r"(tmem_d),
        "r"(tmem_a),
        "r"(desc_lo),
        "r"(desc_hi),
        "r"(idesc),
        "r"(first)
        : "memory");
}

// 16 TMEM lanes x 32 columns from eight halves of mma A-fragments, 4 columns each: regs[2 i], regs[2 i + 1] = {row r, row r + 8 |
// k pair c} of columns 4 i .. 4 i + 3 with r = lane / 4, c = lane % 4
__device__ __forceinline__ void tmem_st_16x128b_x8(uint32_t taddr, const uint32_t (&f)[16])
{
    asm volatile("tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(f[0]),
                 "r"(f[1]), "r"(f[2]), "r"(f[3]), "r"(f[4]), "r"(f[5]), "r"(f[6]), "r"(f[7]), "r"(f[8]), "r"(f[9]), "r"(f[10]), "r"(f[11]),
                 "r"(f[12]), "r"(f[13]), "r"(f[14]), "r"(f[15])
                 : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t* bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// One box of a tensor map -> shared memory, completion counted on an mbarrier
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar)
{
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint64_t* bar)
{
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tc_fence_before()
{
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after()
{
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// sixteen fp32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16])
{
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ uint32_t hmul2_ftz(uint32_t a, uint32_t b)
{
    uint32_t r;
    asm("mul.ftz.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// Bounded wait of a whole warp on a barrier at a shared-memory address; on a time-out the warp records `bit` and plays dead from then on.
__device__ __noinline__ bool wait_on(uint32_t bar, uint32_t parity)
{
    return mbar_wait_warp(reinterpret_cast<uint64_t*>(__cvta_shared_to_generic(bar)), parity);
}
__device__ __forceinline__ void warp_wait(uint32_t bar, uint32_t parity, bool& dead, unsigned* status, unsigned bit)
{
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    // usually the phase is complete already
    if (!__all_sync(0xffffffffu, ok | (dead ? 1u : 0u)) && !wait_on(bar, parity)) {
        if ((threadIdx.x & 31) == 0) atomicOr(status, bit);
        dead = true;
    }
}
__device__ __forceinline__ void arrive_at(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
template<int kOffset>
__device__ __forceinline__ uint4 shared_load16(uint32_t addr)
{
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4+%5];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr), "n"(kOffset) : "memory");
    return v;
}
template<int kOffset>
__device__ __forceinline__ uint32_t shared_load4(uint32_t addr)
{
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1+%2];" : "=r"(v) : "r"(addr), "n"(kOffset) : "memory");
    return v;
}

template<bool kWide>
__global__ void __launch_bounds__(kThreads, 1) gemm_s4_f16_tc_kernel(GemmTcParams p, const __grid_constant__ CUtensorMap x_map,
                                                                      const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap q_map)
{
    using S = Shape<kWide>;
    constexpr int kXST = S::kXST, kAST = S::kAST, kACols = S::kACols, accS = S::kAcc;
    extern __shared__ unsigned char smem_dyn[];
    // tiles the tensor core reads must sit on 1024-byte boundaries (the swizzle is a function of
    // the address bits)
    const uint32_t raw  = smem_u32(smem_dyn);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* sm   = smem_dyn + (base - raw);

    const int TT      = p.token_tile;             // UMMA N, multiple of 16, <= 128
    const int x_bytes = 2 * TT * 128;             // two K blocks of TT rows x 128 B
    unsigned char* x_ring = sm;                                   // kXST x x_bytes (multiples of 1024)
    unsigned char* w_ring = x_ring + kXST * x_bytes;              // kWST x kWStage
    Bars*          bars   = reinterpret_cast<Bars*>(w_ring + kWST * kWStage);

    const int tid  = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;

    const int t0     = blockIdx.y * 128;
    const int t_rows = min(TT, p.T - t0);

    const int G         = p.K / kGroup;
    const int upc       = p.units_per_cta;
    // Two ways of dealing the (column tile, group) units to the CTAs: `parts` CTAs per column tile, each with up
    // to `upc` consecutive groups of it (no CTA touches two tiles); or, with parts == 0, the flat unit list cut
    // into runs of `upc` (a run may end one tile and begin the next).
    const int parts     = p.parts_per_tile;
    const int u_begin   = parts ? (blockIdx.x / parts) * G + (blockIdx.x % parts) * upc : blockIdx.x * upc;
    const int n_units   = parts ? min(upc, G - (int)(blockIdx.x % parts) * upc) : min(u_begin + upc, p.total_units) - u_begin;
    // the CTAs that share column tile `tile`: first CTA and how many
    auto tile_ctas = [&](int tile, int& c_first) {
        if (parts) {
            c_first = tile * parts;
            return parts;
        }
        c_first = (tile * G) / upc;
        return ((tile + 1) * G - 1) / upc - c_first + 1;
    };

    const int  dw = warp - kDqWarp0;  // 0..15 for the expanding warps
    // A unit's packed weight, four slabs of eight adjacent tiles, and its row of {zero, scale}: a box each (zeros beyond N).  Copies of
    // contiguous pieces, five a unit, kept the loader's lane busy for longer than the expansion takes.
    auto w_load = [&](int js, int g, int stage) {
        const uint32_t dst = base + (uint32_t)(w_ring - sm) + (uint32_t)stage * kWStage;
        mbar_arrive_expect_tx(&bars->w_full[stage], (uint32_t)kWStage);
        tma_load_3d(dst, &w_map, 0, js * (kSuperN / 32), g * kSlabs, &bars->w_full[stage]);
        tma_load_2d(dst + kSlabs * kSlabBytes, &q_map, js * kSuperN, g, &bars->w_full[stage]);
    };
    int w_js = u_begin / G, w_g = u_begin - w_js * G;  // the weight loader's next unit
    auto w_next = [&]() {
        if (++w_g == G) w_g = 0, ++w_js;
    };
    if (warp == kWLoadWarp) {
        // The first copies start at once, ahead of the TMEM set-up (one stage: issuing them all takes longer than that) and, unless the
        // kernel before may write the packed weight, of the wait for it.
        if (elect_one()) {
            for (int s = 0; s < kWST; ++s) {
                mbar_init(&bars->w_full[s], 1);
                mbar_init(&bars->w_empty[s], kDqWarps / 2);
            }
            fence_mbar_init();
            if (p.late_weight) pdl_wait();
            w_load(w_js, w_g, 0);
        }
        __syncwarp();
        w_next();
    }

    if (tid == 0) {
        for (int m = 0; m < kTeams; ++m) {
            for (int s = 0; s < kASTMax; ++s) {
                mbar_init(&bars->a_full[m][s], kTeamWarps / 2);
                mbar_init(&bars->a_empty[m][s], 1);
            }
            mbar_init(&bars->acc_full[m], 1);
            mbar_init(&bars->acc_empty[m], kTeamWarps);
        }
        for (int s = 0; s < kXSTMax; ++s) {
            mbar_init(&bars->x_full[s], 1);
            mbar_init(&bars->x_empty[s], kTeams);
        }
        fence_mbar_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)),
                     "n"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem   = bars->tmem_base;
    const uint32_t a_base = tmem + kTeams * accS;  // first expanded-weight stage

    if (warp == 0) {
        // ================================================================== activation loader
        // slice [TT tokens][128 k] of a group -> two 64-wide K blocks, rows of 128 B with their 16-byte
        // chunks XOR-swizzled by (row & 7): the layout the tensor core expects and the one a tensor-map
        // copy with 128-byte swizzle writes.  One slice serves both feature tiles of the unit.
        if (elect_one()) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&x_map)) : "memory");
        __syncwarp();
        pdl_wait();  // the activations come from the kernel before this one
        pdl_launch_dependents();
        if (elect_one()) {
            int g = u_begin % G, it = 0, st = 0;
            for (uint32_t ph = 1; it < n_units; ++it) {  // (a fresh barrier counts as having completed the phase before)
                if (!mbar_wait(&bars->x_empty[st], ph)) {
                    atomicOr(p.status, kStatusGemmPipeWait);
                    break;
                }
                mbar_arrive_expect_tx(&bars->x_full[st], (uint32_t)x_bytes);
                tma_load_3d(base + (uint32_t)(x_ring - sm) + st * x_bytes, &x_map, 0, t0, 2 * g, &bars->x_full[st]);
                if (++g == G) g = 0;
                if (++st == kXST) st = 0, ph ^= 1;
            }
            // this CTA's shared memory may not be left while copies are on their way into it
            for (int i = max(0, it - kXST); i < it; ++i) mbar_wait(&bars->x_full[i % kXST], (i / kXST) & 1);
        }
        __syncwarp();
    }
    else if (warp == kWLoadWarp) {
        // ================================================================== loader of the packed weight
        if (elect_one()) {
            int it = 1, st = 1;
            for (uint32_t ph = 1; it < n_units; ++it) {
                if (!mbar_wait(&bars->w_empty[st], ph)) {
                    atomicOr(p.status, kStatusGemmPipeWait);
                    break;
                }
                w_load(w_js, w_g, st);
                w_next();
                if (++st == kWST) st = 0, ph ^= 1;
            }
            for (int i = max(0, it - kWST); i < it; ++i) mbar_wait(&bars->w_full[i % kWST], (i / kWST) & 1);
        }
        __syncwarp();
    }
    else if (warp <= kIssuers) {
        // ================================================================== MMA issuers
        // One elected lane per team runs the whole loop: waits, eight MMAs, commits.  What it does between two units is a chain that
        // nothing hides, so the team is a constant (operands in uniform registers) and no vote stands in the loop: a unit took 1100
        // cycles of this lane, whatever the tokens, where the tensor core needs 16 x (6 + tokens / 2).
        auto issue = [&](auto team) {
            constexpr int m = decltype(team)::value;
            if (!elect_one()) return;
            const uint32_t idesc   = (1u << 4) | ((uint32_t)(TT >> 3) << 17) | ((uint32_t)(kTileN >> 4) << 24);
            const uint32_t d_tmem  = tmem + m * accS;
            const uint32_t kb_step = (uint32_t)(TT * 128) >> 4;  // descriptor units (16 B) between the two K blocks
            const uint64_t d_ring  = make_desc(base + (uint32_t)(x_ring - sm));
            const uint32_t d_hi    = (uint32_t)(d_ring >> 32);
            // (the low word of the descriptor carries the address: 14 bits of 16-byte units, never a carry out)
            const uint32_t d_lo    = (uint32_t)d_ring;
            const uint32_t x_step  = (uint32_t)x_bytes >> 4;
            int  seg_idx = 0;
            bool first   = true;  // first MMA of the current segment overwrites the accumulator
            int  g       = u_begin % G;
            int  sa = 0, sx = 0;
            uint32_t pa = 0, px = 0;  // phase parity of the weight / activation rings
            for (int it = 0; it < n_units; ++it) {
                bool ok = true;
                if (first && seg_idx > 0) {
                    // the epilogue of the previous segment must have drained the accumulators
                    ok = mbar_wait(&bars->acc_empty[m], (seg_idx - 1) & 1);
                }
                ok = ok && mbar_wait(&bars->x_full[sx], px);
                const bool     last = (it == n_units - 1) || (g == G - 1);
                const uint32_t lo   = d_lo + (uint32_t)sx * x_step;
#pragma unroll
                for (int part = 0; part < S::kParts; ++part) {
                    ok = ok && mbar_wait(&bars->a_full[m][sa], pa);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t a_tmem = a_base + (m * kAST + sa) * kACols;
                    umma_f16_ts_x4(d_tmem, a_tmem, lo + part * kb_step, d_hi, idesc, part == 0 && first ? 1u : 0u);
                    if (S::kParts == 1) umma_f16_ts_x4(d_tmem, a_tmem + 32, lo + kb_step, d_hi, idesc, 0u);
                    umma_commit(&bars->a_empty[m][sa]);
                    if (++sa == kAST) sa = 0, pa ^= 1;
                }
                if (!ok) {
                    atomicOr(p.status, kStatusGemmPipeWait);
                    break;
                }
                umma_commit(&bars->x_empty[sx]);
                first = last;
                if (last) {
                    umma_commit(&bars->acc_full[m]);
                    ++seg_idx;
                }
                if (++g == G) g = 0;
                if (++sx == kXST) sx = 0, px ^= 1;
            }
        };
        if (warp == 1) {
            issue(Int<0>{});
        }
        else {
            issue(Int<1>{});
        }
        __syncwarp();
    }
    else {
        // ================================================================== expand + epilogue
        const int  m    = dw >> 3;        // team = 128-feature tile of the unit
        const int  q    = warp & 3;       // TMEM lane quarter this warp may access = its 32-feature tile
        const int  kh   = (dw >> 2) & 1;  // which of two units it expands (what a unit costs beside the words is shared by
                                          // twice as many), and which half of the token columns it drains
        const int  r    = lane >> 2;
        bool       dead = false;
        int        seg_idx = 0;
        const int  dtid = tid - kDqWarp0 * 32;

        // split-K: [slot][TT tokens][256 feature rows] fp32 partial tiles (a warp touches 128 contiguous
        // bytes per token: whole sectors), per tile a count of CTAs whose partial is complete and a count of
        // CTAs that are done reading.  Tiles this CTA shares with others are reduced after its last unit.
        const size_t slot_floats = (size_t)kSuperN * TT;
        float* const slots  = p.workspace + (size_t)blockIdx.y * p.slots_per_chunk * slot_floats;
        int* const   arrive = p.counters + (size_t)blockIdx.y * p.n_col_tiles;
        int* const   done   = p.counters + (size_t)(gridDim.y + blockIdx.y) * p.n_col_tiles;
        constexpr int kMaxPending = 4;
        int           pend[kMaxPending] = {0, 0, 0, 0};
        int           n_pend = 0;
        // producer side of a folded norm: sums of squares of this CTA's share, [token][quad of features], until a thread for each token adds
        // them up.  In a place of their own: no ring may be written while the other team's products may be reading it.
        float* s_ssq = reinterpret_cast<float*>(bars + 1);
        // Outputs of four adjacent features of a token from their sum
        auto finish = [&](int t, int quad, int col, float4 acc, uint2 res, uint2 gain, float scale) {
            if (p.norm.ssq_in) acc.x *= scale, acc.y *= scale, acc.z *= scale, acc.w *= scale;
            const __half2 h0 = __floats2half2_rn(acc.x, acc.y), h1 = __floats2half2_rn(acc.z, acc.w);
            auto half2_of    = [](uint32_t v) { return __half22float2(reinterpret_cast<const __half2&>(v)); };
            auto word_of     = [](__half2 v) { return reinterpret_cast<const uint32_t&>(v); };
            if (p.norm.ssq_out) {
                // producer side (llama_decoder_kernels.cu:104-160 split in two): residual += y in fp32, stored as
                // fp16; the sum of squares is taken before that rounding, the norm weight applied to the stored value
                const float2  r0 = half2_of(res.x), r1 = half2_of(res.y);
                const float2  y0 = __half22float2(h0), y1 = __half22float2(h1);
                const float2  s0 = make_float2(r0.x + y0.x, r0.y + y0.y), s1 = make_float2(r1.x + y1.x, r1.y + y1.y);
                const float   ss = (s0.x * s0.x + s0.y * s0.y) + (s1.x * s1.x + s1.y * s1.y);
                const __half2 n0 = __float22half2_rn(s0), n1 = __float22half2_rn(s1);
                const size_t  at = (size_t)(t0 + t) * p.N + col;
                *reinterpret_cast<uint2*>(p.norm.residual + at) = make_uint2(word_of(n0), word_of(n1));
                const float2 a0 = __half22float2(n0), a1 = __half22float2(n1);
                float2       g0 = half2_of(gain.x), g1 = half2_of(gain.y);
                g0.x *= scale, g0.y *= scale, g1.x *= scale, g1.y *= scale;  // a power of two
                *reinterpret_cast<uint2*>(p.C + at) =
                    make_uint2(word_of(__floats2half2_rn(a0.x * g0.x, a0.y * g0.y)), word_of(__floats2half2_rn(a1.x * g1.x, a1.y * g1.y)));
                s_ssq[t * kSquaresLd + quad] = ss;
            }
            else if (p.fused_silu) {
                // kernels/gemm_s_f16/gemm_s4_f16.cu:31-43 on the fp16-rounded pairs (gate, up)
                const float2 u0 = __half22float2(h0), u1 = __half22float2(h1);
                const float  s0 = u0.x / (1.f + __expf(-u0.x)), s1 = u1.x / (1.f + __expf(-u1.x));
                *reinterpret_cast<__half2*>(p.C + (size_t)(t0 + t) * (p.N / 2) + col / 2) = __floats2half2_rn(s0 * u0.y, s1 * u1.y);
            }
            else {
                *reinterpret_cast<uint2*>(p.C + (size_t)(t0 + t) * p.N + col) = make_uint2(word_of(h0), word_of(h1));
            }
        };
        // Rows [f0, f1) of a tile, summed over its partials in CTA order.  A thread takes kPieces pieces of four features at a time and
        // asks for kParts partials of each together: eight loads on their way, whatever the number of parts.
        auto sum_rows = [&](auto pieces_of, auto parts_of, auto residual_of, const float* tile_slots, int n_split, int f0, int f1, int col0) {
            constexpr int  kPieces = decltype(pieces_of)::value, kParts = decltype(parts_of)::value;
            constexpr bool kResidual = decltype(residual_of)::value != 0;
            const unsigned quads = (unsigned)(f1 - f0) / 4, items = (unsigned)t_rows * quads;
            const unsigned magic = quads > 1 ? 0xffffffffu / quads + 1 : 0;  // i / quads for i < 2^16: the upper word of i * magic
            for (unsigned i0 = dtid; i0 < items; i0 += kPieces * kDqThreads) {
                float4 acc[kPieces];
                uint2  res[kPieces], gain[kPieces];
                int    tt[kPieces], nn[kPieces];
#pragma unroll
                for (int j = 0; j < kPieces; ++j) {
                    const unsigned i = min(i0 + j * kDqThreads, items - 1);
                    tt[j]  = quads > 1 ? (int)__umulhi(i, magic) : (int)i;
                    nn[j]  = f0 + ((int)i - tt[j] * (int)quads) * 4;
                    acc[j] = make_float4(0.f, 0.f, 0.f, 0.f);
                    res[j] = gain[j] = make_uint2(0u, 0u);
                    if (kResidual && p.norm.ssq_out) {
                        const uint32_t* g = reinterpret_cast<const uint32_t*>(p.norm.norm_weight + col0 + nn[j]);
                        res[j]  = *reinterpret_cast<const uint2*>(p.norm.residual + (size_t)(t0 + tt[j]) * p.N + col0 + nn[j]);
                        gain[j] = make_uint2(__ldg(g), __ldg(g + 1));
                    }
                }
                for (int cc = 0; cc < n_split; cc += kParts) {
                    float4 part[kPieces][kParts];
#pragma unroll
                    for (int j = 0; j < kPieces; ++j) {
                        const float* src = tile_slots + (size_t)cc * slot_floats + tt[j] * kSuperN + nn[j];
#pragma unroll
                        for (int e = 0; e < kParts; ++e) {
                            part[j][e] = make_float4(0.f, 0.f, 0.f, 0.f);  // an absent slot adds +0
                            if (cc + e < n_split) part[j][e] = __ldcg(reinterpret_cast<const float4*>(src + (size_t)e * slot_floats));
                        }
                    }
#pragma unroll
                    for (int j = 0; j < kPieces; ++j) {
#pragma unroll
                        for (int e = 0; e < kParts; ++e) acc[j].x += part[j][e].x, acc[j].y += part[j][e].y, acc[j].z += part[j][e].z, acc[j].w += part[j][e].w;
                    }
                }
#pragma unroll
                for (int j = 0; j < kPieces; ++j) {
                    if (i0 + j * kDqThreads < items) finish(tt[j], (nn[j] - f0) / 4, col0 + nn[j], acc[j], res[j], gain[j], p.norm.ssq_in || p.norm.ssq_out ? bars->row_scale[tt[j]] : 1.f);
                }
            }
        };
        // Every CTA of a split tile reduces its own share of the feature rows, once all partials of the
        // tile are in scratch: nobody reads more than one tile's worth, and the sum runs in CTA order.
        // p.last_sums: the CTA whose partial is the last one reduces all rows, and nobody waits.
        auto reduce_share = [&](int tjs) {
            int       c_first;
            const int n_split = tile_ctas(tjs, c_first);
            const int col0    = tjs * kSuperN;
            if (dtid == 0 && !p.last_sums) {
                // Bounded wait for the other CTAs of the tile.  The plan splits tiles between CTAs only
                // when the whole grid is one wave of at most one CTA per SM (gemm_tc_plan), so the
                // partners are running or waiting for an SM that a kernel ahead in the stream still
                // holds; that kernel does not depend on this one.
                int             seen = 0;
                const long long t_begin = clock64();
                for (;;) {
                    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(seen) : "l"(arrive + tjs) : "memory");
                    if (seen >= n_split || clock64() - t_begin > p.max_wait_cycles) break;
                    __nanosleep(32);
                }
                if (seen < n_split) atomicOr(p.status, kStatusGemmTmemWait);
                bars->flag = seen >= n_split;
            }
            named_bar_sync(1, kDqThreads);
            const bool tile_ok = p.last_sums || bars->flag != 0;  // read between the barriers: the next call may rewrite the flag
            int through = 0;
            if (dtid == 0 && !p.last_sums) {
                // looked at behind the sums; a CTA that gave up has seen no full count that says that its own has arrived
                if (!tile_ok) __threadfence();
                through = atomicAdd(done + tjs, 1);
                if (!tile_ok) __threadfence();
            }
            const int j      = blockIdx.x - c_first;
            const int n_cols = min(kSuperN, p.N - col0);  // N % 32 == 0
            const int f0     = p.last_sums ? 0 : (n_cols * j / n_split) & ~3;
            const int f1     = p.last_sums || j == n_split - 1 ? n_cols : ((n_cols * (j + 1) / n_split) & ~3);
            if (tile_ok) {
                const float* tile_slots = slots + (size_t)(c_first + tjs) * slot_floats;
                if (f1 > f0) {
                    if (n_split <= 2 && !p.norm.ssq_out) sum_rows(Int<4>{}, Int<2>{}, Int<0>{}, tile_slots, n_split, f0, f1, col0);
                    else if (n_split <= 4) sum_rows(Int<2>{}, Int<4>{}, Int<1>{}, tile_slots, n_split, f0, f1, col0);
                    else sum_rows(Int<1>{}, Int<8>{}, Int<1>{}, tile_slots, n_split, f0, f1, col0);
                }
            }
            named_bar_sync(1, kDqThreads);  // everyone is done reading; the flag may be reused
            if (p.norm.ssq_out && tile_ok && dtid < t_rows && f1 > f0) {
                float ss = 0.f;
                for (int i0 = 0; i0 < (f1 - f0) / 4; i0 += 8) {
                    float part[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) part[i] = i0 + i < (f1 - f0) / 4 ? s_ssq[dtid * kSquaresLd + i0 + i] : 0.f;
#pragma unroll
                    for (int i = 0; i < 8; ++i) ss += part[i];
                }
                add_row_squares(p.norm.ssq_out + t0 + dtid, ss, bars->row_scale[dtid]);
            }
            if (dtid == 0 && p.last_sums) arrive[tjs] = 0;
            if (dtid == 0 && !p.last_sums && through == n_split - 1) {
                // the last CTA through the wait resets both counts for the next launch; one that gave up counts too, so the counts
                // recover after a time-out
                arrive[tjs] = 0;
                done[tjs]   = 0;
            }
        };

        const int      ccount = TT / 2;                      // token columns per warp: [kh * ccount, +ccount)
        const int      n_row  = m * kTileN + q * 32 + lane;  // feature row of the CTA tile held by this thread
        const uint32_t a_lane = (uint32_t)(q * 32) << 16;    // TMEM lanes of this warp

        // shared-memory addresses: this warp's share of a stage of packed weight (a 32-feature tile of each slab) and of {zero, scale},
        // and the barriers of its rings
        const uint32_t my_w = base + (uint32_t)(w_ring - sm) + (uint32_t)((m * 4 + q) * kTileBytes + lane * 16);
        const uint32_t my_q = base + (uint32_t)(w_ring - sm) + (uint32_t)(kSlabs * kSlabBytes + (m * 4 + q) * 128 + r * 4);
        const uint32_t w_full = smem_u32(bars->w_full), w_empty = smem_u32(bars->w_empty);
        const uint32_t a_full = smem_u32(bars->a_full[m]), a_empty = smem_u32(bars->a_empty[m]);
        int      js = u_begin / G, g = u_begin - js * G;
        int      u  = kh;           // this warp's next unit: every other one
        int      sw = kh, sa = kh * S::kParts;  // its stages of packed and of expanded weight, and their phase parities
        uint32_t pw = 0, pa = 0;
        for (int it = 0; it < n_units;) {
            const int this_js = js;
            const int seg_end = it + min(G - g, n_units - it);
            for (; u < seg_end; u += 2) {
                warp_wait(w_full + sw * 8, pw, dead, p.status, kStatusGemmPipeWait);
                const uint32_t wa = my_w + sw * kWStage, qa = my_q + sw * kWStage;
                const uint32_t qv[4]     = {shared_load4<0>(qa), shared_load4<32>(qa), shared_load4<64>(qa), shared_load4<96>(qa)};
                const uint4    w[kSlabs] = {shared_load16<0>(wa), shared_load16<kSlabBytes>(wa), shared_load16<2 * kSlabBytes>(wa),
                                            shared_load16<3 * kSlabBytes>(wa)};
                uint32_t z1024[2], nz64[2], s_lo[2], s_hi[2];
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    const __half2 q_lo = reinterpret_cast<const __half2&>(qv[2 * a]);
                    const __half2 q_hi = reinterpret_cast<const __half2&>(qv[2 * a + 1]);
                    const __half2 zl2  = __half2half2(__hadd(__low2half(q_lo), __float2half_rn(960.f)));
                    const __half2 zh2  = __half2half2(__hneg(__low2half(q_hi)));
                    const __half2 sl2  = __half2half2(__high2half(q_lo));
                    const __half2 sh2  = __half2half2(__high2half(q_hi));
                    z1024[a] = reinterpret_cast<const uint32_t&>(zl2);
                    nz64[a]  = reinterpret_cast<const uint32_t&>(zh2);
                    s_lo[a]  = reinterpret_cast<const uint32_t&>(sl2);
                    s_hi[a]  = reinterpret_cast<const uint32_t&>(sh2);
                }
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    // two slabs: all fragments first (independent chains the scheduler can interleave), then the stores
                    uint32_t f[2][16];  // [16-row half][pieces of 4 columns]
#pragma unroll
                    for (int kk = 0; kk < 2; ++kk) {
                        const uint4    v     = w[2 * half + kk];
                        const uint32_t wv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int wi = 0; wi < 4; ++wi) {
                            const int a = wi & 1, at = kk * 8 + (wi >> 1) * 4;
                            uint32_t  fr[4];
                            unpack_s4_minus_zero(wv[wi], z1024[a], nz64[a], fr);
                            f[a][at]     = hmul2_ftz(fr[0], s_lo[a]);
                            f[a][at + 1] = hmul2_ftz(fr[1], s_hi[a]);
                            f[a][at + 2] = hmul2_ftz(fr[2], s_lo[a]);
                            f[a][at + 3] = hmul2_ftz(fr[3], s_hi[a]);
                        }
                    }
                    if (half == 0) {
                        // everyone in the warp holds its words: the stage may be filled again
                        __syncwarp();
                        if (lane == 0) arrive_at(w_empty + sw * 8);
                    }
                    const bool begins = half == 0 || S::kParts == 2, ends = half == 1 || S::kParts == 2;  // of a TMEM stage
                    if (begins) {
                        // the tensor core must be done with what this TMEM stage held kAST stages ago (the first round passes at
                        // once: a fresh barrier counts as having completed the phase before)
                        warp_wait(a_empty + sa * 8, pa ^ 1u, dead, p.status, kStatusGemmPipeWait);
                        tc_fence_after();
                    }
                    // rows q*32 + a*16 .. +15 (TMEM lanes), k = 64 half .. +63 (32 columns)
                    const uint32_t a_tmem = a_base + (m * kAST + sa) * kACols + a_lane + (begins ? 0u : 32u);
                    tmem_st_16x128b_x8(a_tmem, f[0]);
                    tmem_st_16x128b_x8(a_tmem + (16u << 16), f[1]);
                    if (ends) {
                        // expanded tile visible to the tensor core
                        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) arrive_at(a_full + sa * 8);
                        if (half == 0) {
                            ++sa;  // the unit's second stage; kAST is even then
                        }
                        else {
                            sa += 1 + S::kParts;  // past the other warps' unit
                            if (sa >= kAST) sa -= kAST, pa ^= 1u;
                        }
                    }
                }
                sw += 2;
                if (sw >= kWST) sw -= kWST, pw ^= 1u;
            }
            it = seg_end;
            if (js == u_begin / G) {
                // What follows reads and writes scratch, tickets and the output, which the kernel before this one may still be using.
                pdl_wait();
                // the tokens' factors, under the last products; read behind a barrier of these threads (reduce_share)
                if (const int t = kDqThreads - 1 - dtid; (p.norm.ssq_in || p.norm.ssq_out) && t < t_rows) {
                    const RowSquares r = load_row_squares((p.norm.ssq_in ? p.norm.ssq_in : p.norm.ssq_before) + t0 + t);
                    bars->row_scale[t] = p.norm.ssq_in ? norm_row_scale(p.norm, r) : norm_row_down(p.norm, r);
                    if (p.norm.ssq_out && blockIdx.x == 0) p.norm.ssq_out[t0 + t].exponent = exponent_of_down(bars->row_scale[t]);
                }
            }
            g = 0;
            ++js;

            // ---- 256-feature tile this_js finished for this CTA: drain the accumulators -----------
            int       c_first;
            const int n_split = tile_ctas(this_js, c_first);
            const int col0    = this_js * kSuperN;
            warp_wait(smem_u32(&bars->acc_full[m]), seg_idx & 1, dead, p.status, kStatusGemmTmemWait);
            tc_fence_after();
            const int n_glob = col0 + n_row;
            const uint32_t my_acc = tmem + m * accS + ((uint32_t)(q * 32) << 16);
            if (!dead) {
                float* mine = slots + (size_t)(blockIdx.x + this_js) * slot_floats + n_row;
                for (int cb = 0; cb < ccount; cb += 16) {
                    // sixteen token columns of this thread's feature row (eight, twice, where ccount is not a
                    // multiple of 16: the second half then repeats columns the other warp owns and is dropped)
                    const int col = kh * ccount + cb;
                    float     v[16];
                    tmem_ld16(my_acc + (uint32_t)col, v);
                    const int valid = min(16, ccount - cb);  // 8 or 16
                    if (n_split > 1) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            if (i < valid) __stcg(mine + (size_t)(col + i) * kSuperN, v[i]);
                        }
                    }
                    else {
                        if (p.norm.ssq_in) {
                            const float mine = norm_row_scale(p.norm, load_row_squares(p.norm.ssq_in + t0 + min(col + (lane & 15), t_rows - 1)));
#pragma unroll
                            for (int i = 0; i < 16; ++i) v[i] *= __shfl_sync(0xffffffffu, mine, i);
                        }
                        // Neighbouring lanes trade a token each, so that a lane holds two adjacent features of one token of every two: whole
                        // sectors, and (gate, up) side by side (22016 x 4096, 735 tokens: 129 us with a store of 2 bytes for every value, 114 so).
                        const bool odd = lane & 1;
                        const int  n0  = n_glob & ~1, tl = t0 + col + odd;
                        const bool in  = n0 < p.N;
                        __half*    out = p.fused_silu ? p.C + (size_t)tl * (p.N / 2) + n0 / 2 : p.C + (size_t)tl * p.N + n0;
                        const int  ld  = p.fused_silu ? p.N : 2 * p.N;  // two tokens
#pragma unroll
                        for (int i = 0; i < 16; i += 2) {
                            const float   got = __shfl_xor_sync(0xffffffffu, odd ? v[i] : v[i + 1], 1);
                            const __half2 h   = odd ? __floats2half2_rn(got, v[i + 1]) : __floats2half2_rn(v[i], got);
                            if (in && i < valid && tl + i < p.T) {
                                if (p.fused_silu) {
                                    // kernels/gemm_s_f16/gemm_s4_f16.cu:31-43 on the fp16-rounded pair (gate, up)
                                    const float2 u = __half22float2(h);
                                    *out = __float2half_rn(u.x / (1.f + __expf(-u.x)) * u.y);
                                }
                                else {
                                    *reinterpret_cast<__half2*>(out) = h;
                                }
                            }
                            out += ld;
                        }
                    }
                }
            }
            ++seg_idx;
            // the accumulators may be overwritten now
            tc_fence_before();
            __syncwarp();
            if (lane == 0 && !dead) mbar_arrive(&bars->acc_empty[m]);
            if (n_split > 1) {
                // Publish the partial (its reduction waits until this CTA has no units left): the barrier orders every thread's stores before
                // the release of the one thread that then counts the CTA in.  (Each warp counting itself in: sixteen releases instead of one,
                // 4096 x 4096 with 16 / 32 / 64 / 128 tokens 8.1 / 8.8 / 9.8 / 13.2 us, 7.8 / 8.2 / 9.2 / 12.4 so; 4096 x 11008 with 64
                // 14.4 and 13.8.)
                named_bar_sync(1, kDqThreads);
                if (!p.last_sums && dtid == 0) asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(arrive + this_js) : "memory");
                if (p.last_sums) {
                    if (dtid == 0) {
                        __threadfence();
                        const int before = atomicAdd(arrive + this_js, 1);
                        __threadfence();
                        bars->flag = before == n_split - 1;
                    }
                    named_bar_sync(1, kDqThreads);
                    if (bars->flag == 0) continue;  // rewritten behind the next barrier of these threads at the earliest
                }
                if (n_pend == kMaxPending) {
                    reduce_share(pend[0]);
                    for (int i = 1; i < kMaxPending; ++i) pend[i - 1] = pend[i];
                    --n_pend;
                }
                pend[n_pend++] = this_js;
            }
        }
        for (int i = 0; i < n_pend; ++i) {
            reduce_share(pend[i]);
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(kTmemCols) : "memory");
    }
}

using PFN_encodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                     const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                     CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// the driver's tensor-map encoder, found through the runtime so that the library does not link libcuda
PFN_encodeTiled lookup_encode_tiled()
{
    void*                           fn = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess
        || q != cudaDriverEntryPointSuccess) {
        return nullptr;
    }
    return reinterpret_cast<PFN_encodeTiled>(fn);
}

}  // namespace

size_t gemm_tc_smem_bytes(int token_tile)
{
    return 1024 + (size_t)(token_tile > 64 ? Shape<true>::kXST : Shape<false>::kXST) * 2 * token_tile * 128 + (size_t)kWST * kWStage + sizeof(Bars)
           + (size_t)token_tile * kSquaresLd * sizeof(float) + 64;
}

GemmTcPlan gemm_tc_plan(int N, int T, int K, int sm_count, bool balance)
{
    GemmTcPlan pl{};
    pl.token_tile  = T >= 128 ? 128 : ((T + 15) / 16) * 16;
    pl.t_chunks    = (T + 127) / 128;
    pl.n_col_tiles = (N + kSuperN - 1) / kSuperN;
    const int G    = K / kGroup;
    pl.total_units = pl.n_col_tiles * G;
    pl.parts_per_tile = 0;
    // With at least as many whole column tiles as SMs: one per CTA, nothing is split, nobody waits.  `balance`: unless their last
    // wave is so empty that cutting the units evenly is faster, by a model fitted to 70 launches of seven projections with 17 to 1024
    // tokens, both ways (microseconds; mean error 8 % and 4 %; the way it picks costs 1.8 % more than the better one, always whole
    // tiles 5.5 %).  57344 x 8192, 224 tiles: two waves of 64 units, or 97 units for every SM: 71 / 62 us with 32 tokens.
    const long long tiles = (long long)pl.t_chunks * pl.n_col_tiles;
    const double    fill  = std::max(0, pl.token_tile - 32) / 96.0;  // what a unit costs beyond its expansion
    auto cut_us = [&](int units) { return 1.0 + units * (0.547 + 0.409 * fill) + 2.5 * units / G + 3.4 * pl.token_tile / 128; };
    bool whole = tiles >= sm_count;
    const bool could = whole;
    if (whole) {
        pl.us = (double)((tiles + sm_count - 1) / sm_count) * (G * (0.489 + 0.317 * fill) + 3.5);
        if (balance && pl.t_chunks <= sm_count / 2) {
            const int per_chunk = sm_count / pl.t_chunks;
            whole = pl.us <= cut_us((pl.total_units + per_chunk - 1) / per_chunk);
        }
    }
    if (whole) {
        pl.units_per_cta = G;
        pl.ctas          = pl.n_col_tiles;
    }
    else {
        // K is split between CTAs only while the whole grid is a single wave of one CTA per SM: CTAs
        // that share a column tile wait for one another, so all of them must be able to run together
        int ctas = sm_count / pl.t_chunks;
        if (ctas > pl.total_units) ctas = pl.total_units;
        const int flat = (pl.total_units + ctas - 1) / ctas;  // units per CTA when the flat unit list is cut evenly
        // Prefer a whole number of CTAs per column tile when that costs at most one unit more per CTA: a CTA whose
        // run of units crosses from one tile into the next publishes and reduces two partial tiles instead of one.
        const int per_tile = ctas / pl.n_col_tiles;  // 0 where more tiles than CTAs are cut
        const int part     = per_tile >= 2 ? (G + per_tile - 1) / per_tile : G;  // units per CTA with per_tile CTAs on every tile
        if (per_tile >= 2 && part <= flat + 1) {
            pl.parts_per_tile = (G + part - 1) / part;
            pl.units_per_cta  = part;
            pl.ctas           = pl.n_col_tiles * pl.parts_per_tile;
        }
        else {
            pl.units_per_cta = flat;
            pl.ctas          = (pl.total_units + flat - 1) / flat;
        }
        pl.us = cut_us(pl.units_per_cta);
    }
    // Tiles that are cut only because it is faster are summed by the CTA that is done last: a product of that size never depended on
    // its CTAs running together, and loses nothing by it (us, last one / each a share, two runs: 57344 x 8192 with 32 tokens 68, 71 / 74, 72,
    // with 128 108, 110 / 110, 116; 8192 x 28672 with 300 tokens 150, 155 / 155, 152; 4096 x 11008 with 1200 130, 127 / 134, 126).
    // With fewer tiles than SMs every CTA sums a share (4096 x 11008 with 16 / 64 tokens: 11.7 / 13.9 us, by the last one 12.8 / 22.9).
    pl.last_sums       = could && !whole;
    pl.slots_per_chunk = pl.ctas + pl.n_col_tiles;
    pl.smem_bytes      = gemm_tc_smem_bytes(pl.token_tile);
    pl.workspace_floats = pl.units_per_cta % G == 0 ? 0 : (size_t)pl.t_chunks * pl.slots_per_chunk * pl.token_tile * kSuperN;
    pl.counter_ints     = (size_t)2 * pl.t_chunks * pl.n_col_tiles;  // arrivals and finished readers per tile
    return pl;
}

bool gemm_tc_all_tiles_split(const GemmTcPlan& pl, int K)
{
    if (pl.t_chunks != 1) return false;
    if (pl.parts_per_tile) return pl.parts_per_tile >= 2;
    return pl.units_per_cta < K / kGroup && pl.ctas > 1;  // a run of the flat list is shorter than a tile: every tile has several owners
}

cudaError_t gemm_tc_prepare(int max_smem)
{
    const cudaError_t e = cudaFuncSetAttribute(gemm_s4_f16_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(gemm_s4_f16_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
}
static const KernelPreparation g_prepare(gemm_tc_prepare);

cudaError_t gemm_tc_launch(const GemmTcPlan& pl, GemmTcParams p, cudaStream_t st, bool pdl)
{
    p.units_per_cta   = pl.units_per_cta;
    p.parts_per_tile  = pl.parts_per_tile;
    p.total_units     = pl.total_units;
    p.slots_per_chunk = pl.slots_per_chunk;
    p.n_col_tiles     = pl.n_col_tiles;
    p.token_tile      = pl.token_tile;
    p.last_sums       = pl.last_sums;
    if (p.max_wait_cycles <= 0) p.max_wait_cycles = kMaxWaitCycles;

    static const PFN_encodeTiled encode = lookup_encode_tiled();
    if (encode == nullptr) return cudaErrorNotSupported;
    auto map_of = [](CUtensorMap& map, CUtensorMapDataType type, int rank, const void* at, std::array<cuuint64_t, 3> dims,
                     std::array<cuuint64_t, 2> strides, std::array<cuuint32_t, 3> box, CUtensorMapSwizzle swizzle) {
        const cuuint32_t steps[3] = {1u, 1u, 1u};
        return encode(&map, type, rank, const_cast<void*>(at), dims.data(), strides.data(), box.data(), steps, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
               == CUDA_SUCCESS;
    };
    CUtensorMap      x_map, w_map, q_map;
    const cuuint64_t N = p.N, T = p.T, K = p.K;
    // [K / 64][T][64] fp16: a unit's two 64-wide blocks (128 bytes, the swizzle span) of the token tile; [K / 32][N / 32][512 bytes]: four
    // slabs of a column tile; [K / 128][N] {zero, scale}
    if (!map_of(x_map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, p.X, {64, T, K / 64}, {K * 2, 128}, {64u, (cuuint32_t)pl.token_tile, 2u},
                CU_TENSOR_MAP_SWIZZLE_128B)
        || !map_of(w_map, CU_TENSOR_MAP_DATA_TYPE_INT64, 3, p.A, {kTileBytes / 8, N / 32, K / 32}, {kTileBytes, N / 32 * kTileBytes},
                   {kTileBytes / 8, kSuperN / 32, kSlabs}, CU_TENSOR_MAP_SWIZZLE_NONE)
        || !map_of(q_map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, p.Q, {N, K / kGroup, 1}, {N * 4, 0}, {kSuperN, 1u, 1u}, CU_TENSOR_MAP_SWIZZLE_NONE)) {
        return cudaErrorInvalidValue;
    }
    dim3 grid(pl.ctas, pl.t_chunks);
    return launch_kernel(pl.token_tile > 64 ? gemm_s4_f16_tc_kernel<true> : gemm_s4_f16_tc_kernel<false>, grid, dim3(kThreads), pl.smem_bytes, st, pdl, p, x_map, w_map, q_map);
}

}  // namespace tmb
