// The three decode operators over the recurrent kernel: the [B,T,H,D] step, the reference's state-pool step and the KDA step.
#include "runtime.h"

namespace fla_host {

static void activation_ok(const char* op, const char* name, const Tensor& t) {
  // fp16 activations are read exactly by the decode kernel (fp32 arithmetic on CUDA cores); q, k, v share one dtype
  TORCH_CHECK_TYPE(t.scalar_type() == at::kBFloat16 || t.scalar_type() == at::kHalf, op, ": ", name, " dtype must be torch.bfloat16 or torch.float16, got ",
                   t.scalar_type());
}
static Tensor gate(const Tensor& t, const char* op) {      // fp16 gates become fp32
  if (!t.defined() || t.scalar_type() != at::kHalf) return t;
  return convert(t.reshape({-1, t.size(-1)}), at::kFloat, op).view(t.sizes());
}
// [B, T, ...] as [B * T, ...]: a view of the descriptor where the strides allow it, else a copy.
static fla_tensor_t merged(const Tensor& t, Tensor& keep) {
  keep = t;
  const int64_t B = t.size(0), T = t.size(1);
  if (B > 1 && T > 1 && t.stride(0) != T * t.stride(1)) keep = t.contiguous();
  fla_tensor_t d = desc(keep), r = d;
  r.ndim = d.ndim - 1;
  r.shape[0] = B * T;
  r.stride[0] = T > 1 ? d.stride[1] : d.stride[0];
  for (int i = 1; i < r.ndim; ++i) r.shape[i] = d.shape[i + 1], r.stride[i] = d.stride[i + 1];
  r.shape[r.ndim] = r.stride[r.ndim] = 0;
  return r;
}
static void run(const char* op, fla_recurrent_gdn_args& a, at::Device d) {
  two_phase("recurrent_gdn", lib.recurrent_gdn_workspace_size, lib.recurrent_gdn, a, d);
  (void)op;
}

Pair recurrent_fused(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g_, const Tensor& beta_, double scale, const Tensor& h0,
                     bool want_final, bool l2norm, const Tensor& cu_, bool v_first, bool inplace, const Tensor& gk_) {
  const char* op = "fused_recurrent_gated_delta_rule";
  activation_ok(op, "q", q), activation_ok(op, "k", k), activation_ok(op, "v", v);
  TORCH_CHECK_TYPE(q.scalar_type() == k.scalar_type() && k.scalar_type() == v.scalar_type(), op, ": q, k, v must share one dtype, got ", q.scalar_type(), ", ",
                   k.scalar_type(), ", ", v.scalar_type());
  TORCH_CHECK(q.dim() == 4 && q.sizes() == k.sizes() && v.dim() == 4, op, ": q/k must be [B,T,HK,K] and v [B,T,HV,V]");
  const int64_t B = q.size(0), T = q.size(1), HK = q.size(2), K = q.size(3), HV = v.size(2), V = v.size(3);
  TORCH_CHECK(HK > 0 && HV % HK == 0, op, ": HV=", HV, " must be a multiple of HK=", HK);
  TORCH_CHECK_VALUE(std::isfinite(scale), op, ": scale must be finite, got ", scale);
  const at::Device d = Device("recurrent_gdn")(q)(k)(v)(g_)(beta_)(h0)(gk_).get();
  const Tensor g = gate(g_, op), beta = gate(beta_, op), gk = gate(gk_, op);
  Tensor cu;
  int64_t N = B;
  if (cu_.defined()) {
    TORCH_CHECK(B == 1, op, ": cu_seqlens requires batch size 1");
    cu = cu_.to(d, at::kInt);
    N = cu.numel() - 1;
  }
  const int64_t r = v_first ? V : K, c = v_first ? K : V;
  Tensor in;
  if (!h0.defined()) {
    in = at::zeros({N, HV, r, c}, q.options().dtype(at::kFloat));
  } else {
    TORCH_CHECK(h0.sizes() == at::IntArrayRef({N, HV, r, c}), op, ": initial_state shape must be ", at::IntArrayRef({N, HV, r, c}), ", got ", h0.sizes());
    // a copy would receive the update and leave the caller's state pool as it was
    TORCH_CHECK(!inplace || h0.is_contiguous(), op, ": inplace_final_state=True needs a contiguous initial_state, got strides ", h0.strides());
    in = h0.contiguous();
  }
  TORCH_CHECK(!inplace || !h0.defined() || !h0.requires_grad(), op, ": initial_state is updated in place and must not require grad");
  const Tensor out_state = inplace ? in : empty(in.sizes(), in.scalar_type(), d);   // the kernel always streams the state back
  Tensor out = empty(v.sizes(), v.scalar_type(), d);
  Tensor kq, kk, kv, kg, kb, kgk, ko;
  fla_recurrent_gdn_args a{};
  a.q = merged(q, kq), a.k = merged(k, kk), a.v = merged(v, kv), a.out = merged(out, ko);
  if (g.defined()) {
    TORCH_CHECK(g.dim() == 3, op, ": g must be [B,T,HV]");
    a.g = merged(g, kg);
  }
  if (beta.defined()) {
    TORCH_CHECK(beta.dim() == 3, op, ": beta must be [B,T,HV]");
    a.beta = merged(beta, kb);
  }
  if (gk.defined()) {
    TORCH_CHECK(gk.sizes() == at::IntArrayRef({B, T, HV, K}), op, ": gk must be ", at::IntArrayRef({B, T, HV, K}), ", got ", gk.sizes());
    a.gk = merged(gk, kgk);
  }
  a.state_in = desc(in), a.state_out = desc(out_state), a.cu_seqlens = desc(cu);
  a.scale = float(scale), a.tokens_per_seq = int32_t(T), a.state_v_first = v_first, a.use_qk_l2norm = l2norm;
  run(op, a, d);
  if (inplace && h0.defined()) out_state.unsafeGetTensorImpl()->bump_version();
  return {out, want_final || inplace ? out_state : Tensor()};
}

Tensor recurrent_pool(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& state, const Tensor& beta_, double scale,
                      const Tensor& lengths, const Tensor& indices, const Tensor& accepted, const Tensor& g_) {
  const char* op = "recurrent_gated_delta_rule";
  activation_ok(op, "query", q), activation_ok(op, "key", k), activation_ok(op, "value", v), activation_ok(op, "beta", beta_);
  TORCH_CHECK_TYPE(q.scalar_type() == k.scalar_type() && k.scalar_type() == v.scalar_type(), op, ": query, key, value must share one dtype, got ",
                   q.scalar_type(), ", ", k.scalar_type(), ", ", v.scalar_type());
  TORCH_CHECK_TYPE(state.scalar_type() == at::kBFloat16 || state.scalar_type() == at::kFloat, op, ": state dtype must be bfloat16 or float32, got ",
                   state.scalar_type());
  TORCH_CHECK_TYPE(lengths.scalar_type() == at::kInt && indices.scalar_type() == at::kInt, op, ": actual_seq_lengths and ssm_state_indices must be int32");
  TORCH_CHECK(q.dim() == 3 && q.sizes() == k.sizes() && v.dim() == 3 && state.dim() == 4, op,
              ": expected query/key [T,Nk,Dk], value [T,Nv,Dv], state [blocks,Nv,Dv,Dk]");
  const int64_t Nk = q.size(1), Dk = q.size(2), Nv = v.size(1), Dv = v.size(2);
  TORCH_CHECK(state.size(1) == Nv && state.size(2) == Dv && state.size(3) == Dk, op, ": state shape must be (blocks, ", Nv, ", ", Dv, ", ", Dk, "), got ",
              state.sizes());
  TORCH_CHECK(Nk > 0 && Nv % Nk == 0, op, ": Nv must be an integer multiple of Nk, got Nv=", Nv, ", Nk=", Nk, ".");
  TORCH_CHECK(lengths.numel() >= 2, op, ": actual_seq_lengths must contain the prefix entry and at least one sequence length.");
  TORCH_CHECK_VALUE(std::isfinite(scale), op, ": scale must be finite, got ", scale, ".");
  TORCH_CHECK(!state.requires_grad(), op, ": state is updated in place and must not require grad");
  const at::Device d = Device("recurrent_gdn")(q)(k)(v)(g_)(beta_)(state)(lengths)(indices)(accepted).get();
  const Tensor beta = gate(beta_, op), g = gate(g_, op), len = lengths.contiguous();
  Tensor out = empty(v.sizes(), v.scalar_type(), d);
  fla_recurrent_gdn_args a{};
  a.q = desc(q), a.k = desc(k), a.v = desc(v), a.g = desc(g), a.beta = desc(beta), a.out = desc(out);
  a.state_in = a.state_out = desc(state);
  a.cu_seqlens = desc(len), a.cu_is_lengths = 1;      // [prefix, l1, l2, ...]: the kernel adds them up
  a.state_indices = desc(indices), a.num_accepted_tokens = desc(accepted);
  a.scale = float(scale), a.state_v_first = 1;
  run(op, a, d);
  state.unsafeGetTensorImpl()->bump_version();
  return out;
}

Pair recurrent_kda(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g_, const Tensor& beta_, const Tensor& h0, const Tensor& cu,
                   const Tensor& indices, const Tensor& a_log, const Tensor& dt_bias, const Tensor& accepted, double scale, bool inplace,
                   bool l2norm, int64_t gate_mode, int64_t beta_mode, double lower_bound, bool v_first, int64_t seq_num) {
  const char* op = "recurrent_kda";
  const at::Device d = Device("recurrent_gdn")(q)(k)(v)(g_)(beta_)(h0)(cu)(indices)(a_log)(dt_bias)(accepted).get();
  const int64_t T = q.size(1), K = q.size(3), HV = v.size(2), V = v.size(3);
  const Tensor g = gate(g_, op), beta = gate(beta_, op);
  const int64_t r = v_first ? V : K, c = v_first ? K : V;
  const Tensor in = h0.defined() ? h0.contiguous() : at::zeros({seq_num, HV, r, c}, q.options().dtype(at::kFloat));
  const Tensor out_state = inplace ? in : empty(in.sizes(), in.scalar_type(), d);
  Tensor out = empty(v.sizes(), v.scalar_type(), d);
  Tensor kq, kk, kv, kb, kg, ko;
  fla_recurrent_gdn_args a{};
  a.q = merged(q, kq), a.k = merged(k, kk), a.v = merged(v, kv), a.beta = merged(beta, kb), a.gk = merged(g, kg), a.out = merged(out, ko);
  if (gate_mode) a.a_log = desc(a_log), a.dt_bias = desc(dt_bias);
  a.state_in = desc(in), a.state_out = desc(out_state);
  a.cu_seqlens = desc(cu), a.state_indices = desc(indices), a.num_accepted_tokens = desc(accepted);
  a.scale = float(scale), a.lower_bound = float(lower_bound), a.tokens_per_seq = int32_t(T);
  a.state_v_first = v_first, a.use_qk_l2norm = l2norm, a.gate_mode = int32_t(gate_mode), a.beta_mode = int32_t(beta_mode);
  run(op, a, d);
  if (inplace && h0.defined()) out_state.unsafeGetTensorImpl()->bump_version();
  return {out, out_state};
}

}  // namespace fla_host
