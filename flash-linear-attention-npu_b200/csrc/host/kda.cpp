// Chunked Kimi Delta Attention: forward, backward and the autograd node over them.
#include "runtime.h"
#include <torch/csrc/autograd/custom_function.h>

namespace fla_host {

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

KdaResult kda_fwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, const Tensor& h0, const Tensor& a_log,
                  const Tensor& dt_bias, const Geometry& geo, const KdaOptions& o, const Tensor& aqk, const Tensor& akk) {
  const int64_t B = q.size(0), T = q.size(1), K = q.size(3), HV = v.size(2), V = v.size(3);
  const at::Device d = Device("kda_chunk_fwd")(q)(k)(v)(g)(beta)(h0)(a_log)(dt_bias)(aqk)(akk).get();
  KdaResult r;
  r.o = empty({B, T, HV, V}, o.out.value_or(q.scalar_type()), d);
  if (o.want_final) r.ht = empty({geo.N, HV, K, V}, at::kFloat, d);
  if (o.want_gk) r.gk = empty({B, T, HV, K}, at::kFloat, d);
  fla_kda_chunk_fwd_args a{};
  a.q = desc(q), a.k = desc(k), a.v = desc(v), a.g = desc(g), a.beta = desc(beta);
  if (o.gate_mode) a.a_log = desc(a_log), a.dt_bias = desc(dt_bias);
  a.initial_state = desc(h0), a.o = desc(r.o), a.final_state = desc(r.ht), a.gk = desc(r.gk);
  a.cu_seqlens = desc(geo.cu), a.chunk_offsets = desc(geo.co);
  a.aqk = desc(aqk), a.akk = desc(akk);
  a.scale = float(o.scale), a.lower_bound = float(o.lower_bound), a.gate_mode = int32_t(o.gate_mode);
  a.chunk_size = kChunk, a.max_seqlen = int32_t(geo.max_len), a.total_chunks = int32_t(geo.chunks);
  if (o.l2norm) {
    r.q_rstd = empty({B, T, q.size(2)}, at::kFloat, d), r.k_rstd = empty({B, T, q.size(2)}, at::kFloat, d);
    a.q_rstd = desc(r.q_rstd), a.k_rstd = desc(r.k_rstd);
  }
  if (o.keep) {      // the reference's disable_recompute=True: keep the intermediates for the backward instead of recomputing them
    uint64_t bytes = 0;
    ok_or_throw("kda_chunk_saved_size", lib.kda_chunk_saved_size(&a, &bytes));
    r.saved = empty({int64_t(bytes + 1) / 2}, at::kBFloat16, d);
    a.saved = desc(r.saved);
  }
  two_phase("kda_chunk_fwd", lib.kda_chunk_fwd_workspace_size, lib.kda_chunk_fwd, a, d, true);
  return r;
}

std::vector<Tensor> kda_bwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, double scale, const Tensor& h0,
                            const Tensor& do_in, const Tensor& dht_in, const Geometry& geo, GradTypes ty, const Tensor& saved,
                            const Tensor& q_rstd, const Tensor& k_rstd) {
  const int64_t B = q.size(0), T = q.size(1), HK = q.size(2), K = q.size(3), HV = v.size(2), V = v.size(3);
  const at::Device d = Device("kda_chunk_bwd")(q)(k)(v)(g)(beta)(h0)(do_in)(dht_in)(saved).get();
  const Tensor d_o = as_rows(do_in.scalar_type() == at::kBFloat16 ? do_in : convert(do_in, at::kBFloat16, "chunk_kda_bwd"));
  const Tensor dht = dht_in.defined() ? dht_in.to(at::kFloat).contiguous() : dht_in;
  Tensor dq = empty({B, T, HK, K}, ty.q, d), dk = empty({B, T, HK, K}, ty.k, d), dv = empty({B, T, HV, V}, ty.v, d), dg = empty({B, T, HV, K}, ty.g, d),
         dbeta = empty({B, T, HV}, ty.beta, d), dh0;
  if (h0.defined()) dh0 = empty({geo.N, HV, K, V}, at::kFloat, d);
  fla_kda_chunk_bwd_args a{};
  a.q = desc(q), a.k = desc(k), a.v = desc(v), a.g = desc(g), a.beta = desc(beta);
  a.initial_state = desc(h0), a.d_o = desc(d_o), a.dht = desc(dht);
  a.dq = desc(dq), a.dk = desc(dk), a.dv = desc(dv), a.dg = desc(dg), a.dbeta = desc(dbeta), a.dh0 = desc(dh0);
  a.cu_seqlens = desc(geo.cu), a.chunk_offsets = desc(geo.co), a.saved = desc(saved);
  a.q_rstd = desc(q_rstd), a.k_rstd = desc(k_rstd);
  a.scale = float(scale), a.chunk_size = kChunk, a.max_seqlen = int32_t(geo.max_len), a.total_chunks = int32_t(geo.chunks);
  two_phase("kda_chunk_bwd", lib.kda_chunk_bwd_workspace_size, lib.kda_chunk_bwd, a, d, true);
  return {dq, dk, dv, dg, dbeta, dh0};
}

// Saves the inputs, and the forward's operand images when they are kept; otherwise the backward recomputes them.
struct KdaFn : torch::autograd::Function<KdaFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta,
                               const OptTensor& h0_, const OptTensor& cu_, const OptTensor& co_, std::vector<int64_t> geo, double scale, bool want_final,
                               int64_t out, bool keep, bool l2norm) {
    const Tensor h0 = value(h0_), cu = value(cu_), co = value(co_);
    KdaOptions o;
    o.scale = scale, o.want_final = want_final, o.keep = keep, o.l2norm = l2norm;
    if (out >= 0) o.out = at::ScalarType(out);
    KdaResult r = kda_fwd(q, k, v, g, beta, h0, Tensor(), Tensor(), Geometry{cu, co, geo[0], geo[1], geo[2]}, o, Tensor(), Tensor());
    ctx->save_for_backward({q, k, v, g, beta, h0, r.saved, r.q_rstd, r.k_rstd, cu, co});
    auto& m = ctx->saved_data;
    m["geo"] = geo;
    m["scale"] = scale;
    ctx->set_materialize_grads(false);
    if (want_final) return {r.o, r.ht};
    return {r.o};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    auto& m = ctx->saved_data;
    const std::vector<int64_t> geo = m["geo"].toIntVector();
    const Tensor d_o = grads[0].defined() ? grads[0].contiguous() : at::zeros(s[2].sizes(), s[2].options());
    auto kernel_type = [](const Tensor& t) { return t.scalar_type() == at::kBFloat16 ? at::kBFloat16 : at::kFloat; };
    const GradTypes want{kernel_type(s[0]), kernel_type(s[1]), kernel_type(s[2]), kernel_type(s[3]), kernel_type(s[4])};
    auto r = kda_bwd(s[0], s[1], s[2], s[3], s[4], m["scale"].toDouble(), s[5], d_o, grads.size() > 1 ? grads[1] : Tensor(),
                     Geometry{s[9], s[10], geo[0], geo[1], geo[2]}, want, s[6], s[7], s[8]);
    for (int i = 0; i < 5; ++i) r[i] = r[i].to(s[i].scalar_type());
    variable_list out(14);
    for (int i = 0; i < 6; ++i) out[i] = r[i];
    return out;
  }
};

KdaCall kda(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& g_, const Tensor& beta_, const Tensor& h0_, const Tensor& a_log_,
            const Tensor& dt_bias_, const Tensor& cu, KdaOptions o, const Tensor& aqk, const Tensor& akk, bool return_saved) {
  const char* op = "chunk_kda";
  Tensor q = q_, k = k_, v = v_, g = g_, beta = beta_;
  const bool half = q.scalar_type() == at::kHalf || k.scalar_type() == at::kHalf || v.scalar_type() == at::kHalf;
  const std::optional<at::ScalarType> out = o.out;
  if (half) {
    // fp16 tensors (the reference's published 4-stage case is fp16, fla/ops/ascendc/kda/KDA_FORWARD_VALIDATION_REPORT.md:133-146):
    // q, k, v are rounded to the bf16 operands of the tensor-core products by the library's conversion kernel, fp16 gates
    // become fp32, o is computed in fp32 and converted to fp16 once; gradients return through the same conversions
    TORCH_CHECK_TYPE(q.scalar_type() == k.scalar_type() && k.scalar_type() == v.scalar_type(), op, ": q, k, v must share one dtype, got ", q.scalar_type(),
                     ", ", k.scalar_type(), ", ", v.scalar_type());
    TORCH_CHECK_NOT_IMPLEMENTED(!(aqk.defined() && aqk.scalar_type() == at::kHalf) && !(akk.defined() && akk.scalar_type() == at::kHalf), op,
                                ": export_scores takes bf16 or fp32 views");
    q = to_dtype(q, at::kBFloat16, op), k = to_dtype(k, at::kBFloat16, op), v = to_dtype(v, at::kBFloat16, op);
    if (g.scalar_type() == at::kHalf) g = to_dtype(g, at::kFloat, op);
    if (beta.scalar_type() == at::kHalf) beta = to_dtype(beta, at::kFloat, op);
    o.out = at::kFloat;
  }
  for (auto& [name, t] : {std::pair<const char*, const Tensor&>{"q", q}, {"k", k}, {"v", v}})
    TORCH_CHECK_TYPE(t.scalar_type() == at::kBFloat16, op, ": ", name, " must be bfloat16 or float16, got ", t.scalar_type());
  TORCH_CHECK(q.dim() == 4 && q.sizes() == k.sizes() && v.dim() == 4 && v.size(0) == q.size(0) && v.size(1) == q.size(1), op,
              ": expected q,k [B,T,HK,K] and v [B,T,HV,V]");
  const int64_t B = q.size(0), T = q.size(1), HK = q.size(2), K = q.size(3), HV = v.size(2), V = v.size(3);
  TORCH_CHECK(K == 128 && (V == 128 || V == 256), op, ": this build supports K = 128 and V = 128 or 256, got K=", K, ", V=", V);
  TORCH_CHECK(HK > 0 && HV % HK == 0, op, ": HV=", HV, " must be a multiple of HK=", HK);
  const std::array<int64_t, 4> gs{B, T, HV, K};
  const std::array<int64_t, 3> bs{B, T, HV};
  TORCH_CHECK(g.sizes() == at::IntArrayRef(gs) && beta.sizes() == at::IntArrayRef(bs), op, ": g must be ", at::IntArrayRef(gs), " and beta ", at::IntArrayRef(bs));
  const at::Device d = Device(op)(q)(k)(v)(g)(beta)(h0_).get();
  q = as_rows(q), k = as_rows(k), v = as_rows(v), g = as_rows(g), beta = as_rows(beta);
  KdaCall c;
  c.geo = geometry(op, B, T, cu, d);
  Tensor h0 = h0_;
  if (h0.defined()) {
    const std::array<int64_t, 4> hs{c.geo.N, HV, K, V};
    TORCH_CHECK(h0.sizes() == at::IntArrayRef(hs), op, ": initial_state must be ", at::IntArrayRef(hs), ", got ", h0.sizes());
    h0 = h0.to(at::kFloat).contiguous();
  }
  if (at::GradMode::is_enabled() && any_requires_grad({q, k, v, g, beta, h0})) {
    TORCH_CHECK_NOT_IMPLEMENTED(!o.want_gk && !aqk.defined(), op, ": return_gate_cumsum / export_scores are not available on the differentiable path");
    variable_list l = KdaFn::apply(q, k, v, g, beta, opt(h0), opt(c.geo.cu), opt(c.geo.co), std::vector<int64_t>{c.geo.N, c.geo.max_len, c.geo.chunks}, o.scale,
                                   o.want_final, o.out ? int64_t(*o.out) : int64_t(-1), o.keep, o.l2norm);
    c.r.o = l[0];
    if (l.size() > 1) c.r.ht = l[1];
  } else {
    if (o.l2norm && return_saved) {      // the export pass behind it reads the normalised rows
      q = l2norm_fwd(q, 1e-6, std::nullopt).first, k = l2norm_fwd(k, 1e-6, std::nullopt).first;
      o.l2norm = false;
    }
    Tensor a_log, dt_bias;
    if (o.gate_mode) {
      a_log = a_log_.to(at::kFloat).contiguous();
      if (dt_bias_.defined()) dt_bias = dt_bias_.to(at::kFloat).reshape({HV, K}).contiguous();
    }
    o.keep = return_saved;
    c.r = kda_fwd(q, k, v, g, beta, h0, a_log, dt_bias, c.geo, o, aqk, akk);
    if (return_saved) c.q = q, c.k = k, c.v = v, c.beta = beta;
  }
  if (half) c.r.o = to_dtype(c.r.o, out.value_or(at::kHalf), op);
  return c;
}

}  // namespace fla_host
