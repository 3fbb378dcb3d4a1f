// The products of gemm_dense.h with the epilogues that no operator of the C ABI reaches alone, and the plan that each gets.
#include "handle.cu"
#include "gemm_dense.cu"

extern "C" {

struct Call {
    tmb::DenseGemm g;
};

Call* call_new() { return new Call(); }
void  call_free(Call* c) { delete c; }

void set_operands(Call* c, const void* x, const void* x2, int x2_from, int ldx, const void* w, int ldw, int tokens, int n_out, int k)
{
    tmb::DenseGemm& g = c->g;
    g.x = x, g.x2 = x2, g.x2_from = x2_from, g.ldx = ldx, g.w = w, g.ldw = ldw, g.tokens = tokens, g.n_out = n_out, g.k = k;
}
void set_scale(Call* c, const float* ssq, int parts, int stride, float inv_width, float eps, const float* gain)
{
    tmb::DenseEpilogue& e = c->g.ep;
    e.ssq = ssq, e.ssq_parts = parts, e.ssq_stride = stride, e.inv_width = inv_width, e.eps = eps, e.gain = gain;
}
void set_store(Call* c, void* out, int out_ld)
{
    c->g.ep.kind = tmb::DenseKind::kStore, c->g.ep.out = out, c->g.ep.out_ld = out_ld;
}
void set_input(Call* c, void* out, int out_ld, int tanh_lo, int tanh_hi, int split, void* act, int act_ld)
{
    tmb::DenseEpilogue& e = c->g.ep;
    e.kind = tmb::DenseKind::kInput, e.out = out, e.out_ld = out_ld, e.tanh_lo = tanh_lo, e.tanh_hi = tanh_hi, e.split = split, e.act = act, e.act_ld = act_ld;
}
void set_f32_columns(Call* c, float* out, int from, int ld)
{
    c->g.ep.f32_out = out, c->g.ep.f32_from = from, c->g.ep.f32_ld = ld;
}
void set_residual(Call* c, float* residual, int ld, void* cast, int cast_ld, float* ssq_out, int ssq_out_stride, const void* gate, int gate_ld,
                  const float* gate_bias, float mult)
{
    tmb::DenseEpilogue& e = c->g.ep;
    e.kind = tmb::DenseKind::kResidual, e.residual = residual, e.residual_ld = ld, e.cast = cast, e.cast_ld = cast_ld, e.ssq_out = ssq_out;
    e.ssq_out_stride = ssq_out_stride, e.gate = gate, e.gate_ld = gate_ld, e.gate_bias = gate_bias, e.mult = mult;
}

// 1: whole tiles, 2: cut tiles, 3: pairs of CTAs
int route(const Call* c, int sms)
{
    const tmb::Plan plan = tmb::plan_of(c->g, sms, false);
    return plan.pair ? 3 : plan.cut ? 2 : 1;
}
int run(tm_handle* h, const Call* c, void* stream)
{
    return tmb::dense_gemm(h, c->g, false, (cudaStream_t)stream, false);
}
int sm_count(const tm_handle* h) { return h->sm_count; }

}  // extern "C"
