// Per-device state behind the opaque tm_handle of the C ABI.
#pragma once
#include <cuda_fp16.h>

#include "gemm_s4_f16.h"
#include "mmha.h"

namespace tmb {
// The last call that used one of a handle's scratch areas
struct ScratchOrder {
    cudaEvent_t        done   = nullptr;
    unsigned long long stream = 0;  // cudaStreamGetId
    bool               used   = false;
};
enum ScratchArea { kGemmScratch = 0, kAttentionScratch = 1, kScratchAreas = 2 };
}  // namespace tmb

struct tm_handle {
    int                device          = 0;
    int                sm_count        = 0;
    int                max_smem        = 0;
    int                l2_bytes        = 0;
    void*              scratch         = nullptr;  // split-K / split-KV partials
    size_t             scratch_bytes   = 0;
    int*               counters        = nullptr;  // self-resetting arrival tickets
    size_t             counter_ints    = 0;
    void*              attn_scratch    = nullptr;  // split-KV partials of the attention kernel
    size_t             attn_scratch_bytes = 0;
    int*               attn_counters   = nullptr;
    size_t             attn_counter_ints = 0;
    void*              op_buffer       = nullptr;  // device copies and scratch of single operator calls, grown on demand
    size_t             op_buffer_bytes = 0;
    tmb::ScratchOrder  scratch_order[tmb::kScratchAreas];
    unsigned*          status          = nullptr;  // device status word (bounded waits)
    int                last_cuda_error = 0;
    unsigned long long launches        = 0;
    int                mmha_chunk      = 0;  // 0 = automatic; TM_B200_MMHA_CHUNK overrides
    int                mmha_warps      = 0;  // 0 = automatic; TM_B200_MMHA_WARPS (1, 2 or 4) overrides
    int                gemm_tc_min_n   = -1; // token count from which the tcgen05 kernel is used (-1: by the product's size); TM_B200_GEMM_TC_MIN overrides
    int                gemm_wait_cycles = 0; // 0 = default bound of the split-tile wait of the tcgen05 GEMM (option "gemm_wait_cycles")
    int                pdl_direct      = 0;  // option "pdl_direct": direct GEMM / attention calls launch with programmatic serialization too
    int                p2p_allreduce   = 1;  // TM_B200_P2P_ALLREDUCE / option "p2p_allreduce": peer-memory all-reduce + norm in the decode step
    int                fold_norm       = 1;  // TM_B200_FOLD_NORM=0 / option "fold_norm": the decode step keeps residual add + RMSNorm as kernels of their own
    int                lm_head_cublas  = 0;  // TM_B200_LM_HEAD_CUBLAS=1 / option "lm_head_cublas": the decode step's lm-head through cuBLAS (comparison only)
    int                gemv_cols       = 1;  // TM_B200_GEMV_COLS / option "gemv_cols": 0 = the small-token GEMM never uses its column-owner kernel,
                                             // 1 = 32-column strips, 2 = 64-column strips
    int                pdl             = 1;  // TM_B200_PDL=0: the decode driver launches its kernels without programmatic dependent launch
};

namespace tmb {
// lm_head.cu: logits[tokens][ld] (fp32) = x[tokens][hidden] . w[vocab][hidden]^T, fp16 operands, tcgen05
int lm_head_launch(float* logits, int ld, const __half* x, const __half* w, int tokens, int vocab, int hidden, unsigned* status,
                   long long max_wait_cycles, int max_smem, cudaStream_t st, bool pdl, unsigned long long* launches);
// prefill.cu: q (rotated) to [batch][heads][seq_len][128], k (rotated) and v to their cache rows, as the two public writers do one after the other
int prefill_write_qkv(void* q_buf, const void* qkv, const void* bias, const int* padding_offset, const int* history, const int* length, int batch,
                      int seq_len, int tokens, int heads, int kv_heads, float rope_base, void* const* k_cache, void* const* v_cache,
                      size_t cache_offset, int max_seq_len, bool int8, const float* kv_scale, cudaStream_t st);
// A kernel file's per-device attributes (shared-memory limits and the like), set whenever a handle is created: one static
// object of this type per file, so that a handle knows no kernel by name.
struct KernelPreparation {
    explicit KernelPreparation(cudaError_t (*fn)(int max_smem));
};
// Set by the drivers around their launches (per host thread): the kernel launches made through the C ABI on this thread carry the
// programmatic-dependent-launch attribute, and read weights before the kernel ahead is complete.  Direct callers may put any kernel
// in front of ours: ScratchUse::dependent.
extern thread_local int g_pdl;
// ... and whether the W4A16 products alone, inside a driver's call, carry it (as direct calls: ScratchUse::dependent).
extern thread_local bool g_pdl_products;
struct PdlScope {
    explicit PdlScope(int on, bool products = false) { g_pdl = on, g_pdl_products = products; }
    ~PdlScope() { g_pdl = 0, g_pdl_products = false; }
};

// Held by a call around the launches that use the handle's scratch and tickets.  Calls of one stream are in order by themselves; a
// call on another stream than the last one waits for it on the device.  A captured call is not ordered against others (its graph runs
// later, on any stream): whoever can do without scratch should ask in_order().
class ScratchUse {
public:
    ScratchUse(tm_handle* h, cudaStream_t st);
    ~ScratchUse();
    ScratchUse(const ScratchUse&)            = delete;
    ScratchUse& operator=(const ScratchUse&) = delete;
    bool in_order() { return nested_ || !captured(); }
    bool begin(ScratchArea area);  // ahead of the first launch; false: a CUDA call failed
    // A direct call's kernels carry the attribute too, but wait for the kernel ahead before they read anything (late_weight): what
    // they gain is its way out and their own launch (a plain launch of a 6 us kernel takes 8.2 us).  Not into a caller's capture; inside
    // a driver's call the driver says.
    bool dependent() { return h_->pdl != 0 && (nested_ ? g_pdl_products : !captured()); }
    bool hold();                   // all areas, for every call of this host thread on the handle until this object ends

private:
    bool captured();

    tm_handle*   h_;
    cudaStream_t st_;
    bool         nested_, holds_ = false;
    int          captured_ = -1;  // not asked yet: calls without scratch need not
    bool         begun_[kScratchAreas] = {};
    const tm_handle* outer_ = nullptr;
};
// Set by the decode driver around ONE tm_gemm_s4_f16 call whose launch should carry a GemmNormFusion (gemm_s4_f16.h);
// the driver has checked with gemm_can_fuse_norm that the call is a single launch that can carry it.
struct GemmNormFusion;
extern thread_local const GemmNormFusion* g_gemm_fusion;
bool gemm_can_fuse_norm(const tm_handle* h, int m, int n, int k, bool producer);
}  // namespace tmb

