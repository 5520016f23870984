// Chunked gated delta rule: forward, backward and the differentiable operator over them.
#include "runtime.h"
#include <torch/csrc/autograd/custom_function.h>

namespace fla_host {

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

static Tensor state_f32(const Tensor& t) { return t.defined() ? t.to(at::kFloat).contiguous() : t; }

struct GdnShape {
  int64_t B, T, HK, HV, K, V, tiles, seg_bytes;
};
static at::ScalarType piece_type(int i) { return i == GdnSaved::kGam || i >= GdnSaved::kQr ? at::kFloat : at::kBFloat16; }
static fla_tensor_t gdn_desc(const GdnShape& s, int i, void* data) {
  const at::ScalarType t = piece_type(i);
  switch (i) {
    case GdnSaved::kGam: return desc_at(data, t, {s.B, s.T, s.HV});
    case GdnSaved::kX: return desc_at(data, t, {s.tiles * 8192});                          // (I + A)^-1 per chunk: value + residual strips
    case GdnSaved::kS: return desc_at(data, t, {s.tiles * (s.V / 64) * 16384});
    case GdnSaved::kVn: return desc_at(data, t, {s.tiles * (s.V / 64) * 8192});
    case GdnSaved::kP: return desc_at(data, t, {s.tiles * 8768});                          // P tile (16 KB) + the chunk's factor record
    case GdnSaved::kSegM: return desc_at(data, t, {s.seg_bytes / 2});
    case GdnSaved::kQn: case GdnSaved::kKn: return desc_at(data, t, {s.B, s.T, s.HK, s.K});
    default: return desc_at(data, t, {s.B, s.T, s.HK});
  }
}
// Bytes of the pieces this call has, 0: absent.
static std::array<int64_t, GdnSaved::kPieces> piece_bytes(const GdnShape& s, bool save, bool l2norm) {
  std::array<int64_t, GdnSaved::kPieces> r{};
  for (int i = 0; i < GdnSaved::kPieces; ++i) {
    if ((i == GdnSaved::kS || i == GdnSaved::kVn || i == GdnSaved::kP) && !save) continue;
    if (i >= GdnSaved::kQn && !l2norm) continue;
    const fla_tensor_t d = gdn_desc(s, i, nullptr);
    int64_t n = d.dtype == FLA_F32 ? 4 : 2;
    for (int j = 0; j < d.ndim; ++j) n *= d.shape[j];
    r[i] = n;
  }
  return r;
}
static fla_tensor_t& piece_desc(fla_gdn_chunk_fwd_args& a, int i) {
  fla_tensor_t* const p[] = {&a.gam, &a.x_inv, &a.s_img, &a.vn_img, &a.p_img, &a.seg_m, &a.q_norm, &a.k_norm, &a.q_rstd, &a.k_rstd};
  return *p[i];
}

std::tuple<Tensor, Tensor, GdnSaved> gdn_fwd(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& g_, const Tensor& beta_, double scale,
                                             const Tensor& h0_, bool want_final, const Tensor& cu, bool save, std::optional<at::ScalarType> out,
                                             bool l2norm, bool one) {
  const char* op = "chunk_gated_delta_rule";
  for (auto& [name, t] : {std::pair<const char*, const Tensor&>{"q", q_}, {"k", k_}, {"v", v_}})
    TORCH_CHECK_TYPE(t.scalar_type() == at::kBFloat16, op, ": ", name, " must be bfloat16 (fp32 inputs are rejected like in the reference), got ", t.scalar_type());
  TORCH_CHECK(q_.dim() == 4 && q_.sizes() == k_.sizes() && v_.dim() == 4 && v_.size(0) == q_.size(0) && v_.size(1) == q_.size(1), op,
              ": expected q,k [B,T,HK,K] and v [B,T,HV,V], got ", q_.sizes(), ", ", k_.sizes(), ", ", v_.sizes());
  const int64_t B = q_.size(0), T = q_.size(1), HK = q_.size(2), K = q_.size(3), HV = v_.size(2), V = v_.size(3);
  TORCH_CHECK(K == 128 && (V == 128 || V == 256), op, ": this build supports K = 128 and V = 128 or 256, got K=", K, ", V=", V);
  TORCH_CHECK(HK > 0 && HV % HK == 0, op, ": HV=", HV, " must be a multiple of HK=", HK);
  const std::array<int64_t, 3> gs{B, T, HV};
  TORCH_CHECK(g_.sizes() == at::IntArrayRef(gs) && beta_.sizes() == at::IntArrayRef(gs), op, ": g and beta must be [B,T,HV]=", at::IntArrayRef(gs), ", got ", g_.sizes(), ", ", beta_.sizes());
  const at::Device d = Device("gdn_chunk_fwd")(q_)(k_)(v_)(g_)(beta_)(h0_).get();
  const Tensor q = as_rows(q_), k = as_rows(k_), v = as_rows(v_), g = as_rows(g_), beta = as_rows(beta_);
  GdnSaved s;
  s.geo = geometry(op, B, T, cu, d);
  const int64_t N = s.geo.N, tiles = s.geo.chunks * HV;
  if (h0_.defined()) {
    const std::array<int64_t, 4> hs{N, HV, K, V};
    TORCH_CHECK(h0_.sizes() == at::IntArrayRef(hs), op, ": initial_state must be ", at::IntArrayRef(hs), ", got ", h0_.sizes());
  }
  const Tensor h0 = state_f32(h0_);
  Tensor o = empty({B, T, HV, V}, out.value_or(q.scalar_type()), d), ht;
  if (want_final) ht = empty({N, HV, K, V}, at::kFloat, d);
  fla_gdn_chunk_fwd_args a{};
  a.q = desc(q), a.k = desc(k), a.v = desc(v), a.g = desc(g), a.beta = desc(beta);
  a.initial_state = desc(h0), a.o = desc(o), a.final_state = desc(ht);
  a.cu_seqlens = desc(s.geo.cu), a.chunk_offsets = desc(s.geo.co);
  a.scale = float(scale), a.chunk_size = kChunk, a.max_seqlen = int32_t(s.geo.max_len), a.total_chunks = int32_t(s.geo.chunks);
  c10::cuda::CUDAGuard guard(d);
  uint64_t seg_bytes = 0;
  if (save) ok_or_throw("gdn_chunk_segments_size", lib.gdn_chunk_segments_size(&a, &seg_bytes));
  GdnShape shape{B, T, HK, HV, K, V, tiles, int64_t(seg_bytes)};
  const auto bytes = piece_bytes(shape, save, l2norm);
  int64_t total = 0;
  for (int i = 0; i < GdnSaved::kPieces; ++i) {
    s.at[i] = bytes[i] ? total : -1;
    total += (bytes[i] + 255) / 256 * 256;
    if (bytes[i] && !one) {
      const fla_tensor_t t = gdn_desc(shape, i, nullptr);
      s.piece[i] = empty(at::IntArrayRef(t.shape, t.ndim), piece_type(i), d);
    }
  }
  // inference keeps nothing: the workspace goes into the same allocation
  uint64_t ws_bytes = 0;
  const bool ws_inside = one && !save;
  if (one) {
    for (int i = 0; i < GdnSaved::kPieces; ++i)
      if (bytes[i]) piece_desc(a, i) = gdn_desc(shape, i, reinterpret_cast<void*>(uintptr_t(256)));      // (for the query: what is there)
    if (ws_inside) ok_or_throw("gdn_chunk_fwd workspace query", lib.gdn_chunk_fwd_workspace_size(&a, &ws_bytes));
    s.slab = empty({total + int64_t(ws_bytes)}, at::kByte, d);
  }
  for (int i = 0; i < GdnSaved::kPieces; ++i)
    if (bytes[i]) piece_desc(a, i) = one ? gdn_desc(shape, i, static_cast<char*>(s.slab.data_ptr()) + s.at[i]) : desc(s.piece[i]);
  if (ws_inside) {
    ok_or_throw("gdn_chunk_fwd", lib.gdn_chunk_fwd(&a, static_cast<char*>(s.slab.data_ptr()) + total, ws_bytes, current_stream(d)));
    if (check_status) raise_device_status("gdn_chunk_fwd", s.slab.narrow(0, total, int64_t(ws_bytes)));
  } else {
    two_phase("gdn_chunk_fwd", lib.gdn_chunk_fwd_workspace_size, lib.gdn_chunk_fwd, a, d, true);
  }
  return {o, ht, s};
}

std::vector<Tensor> gdn_bwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& beta, const GdnSaved& s, const Tensor& do_in,
                            const Tensor& dht_in, double scale, bool want_dh0, GradTypes ty) {
  const char* op = "chunk_gated_delta_rule_bwd";
  const int64_t B = v.size(0), T = v.size(1), HK = q.defined() ? q.size(2) : s.hk, K = 128, HV = v.size(2), V = v.size(3);
  const at::Device d = Device("gdn_chunk_bwd")(q)(k)(v)(beta)(do_in)(dht_in).get();
  const Tensor d_o = as_rows(do_in.scalar_type() == at::kBFloat16 ? do_in : convert(do_in, at::kBFloat16, op));
  const std::array<int64_t, 4> os{B, T, HV, V}, hs{s.geo.N, HV, K, V};
  TORCH_CHECK(d_o.sizes() == at::IntArrayRef(os), op, ": do must be ", at::IntArrayRef(os), ", got ", d_o.sizes());
  TORCH_CHECK(s.slab.defined() || s.piece[GdnSaved::kS].defined(), op, ": the forward was not run with save_for_backward=True");
  if (dht_in.defined()) TORCH_CHECK(dht_in.sizes() == at::IntArrayRef(hs), op, ": dht must be ", at::IntArrayRef(hs), ", got ", dht_in.sizes());
  const Tensor dht = state_f32(dht_in);
  Tensor dq = empty({B, T, HK, K}, ty.q, d), dk = empty({B, T, HK, K}, ty.k, d), dv = empty(os, ty.v, d), dg = empty({B, T, HV}, ty.g, d),
         dbeta = empty({B, T, HV}, ty.beta, d), dh0;
  if (want_dh0) dh0 = empty(hs, at::kFloat, d);
  fla_gdn_chunk_bwd_args a{};
  const int64_t seg_end = s.at[GdnSaved::kQn] >= 0 ? s.at[GdnSaved::kQn] : s.slab.defined() ? s.slab.numel() : 0;
  const GdnShape shape{B, T, HK, HV, K, V, s.geo.chunks * HV, s.slab.defined() && s.at[GdnSaved::kSegM] >= 0 ? seg_end - s.at[GdnSaved::kSegM] : 0};
  auto piece = [&](GdnSaved::Piece i) {
    if (!s.slab.defined()) return desc(s.piece[i]);
    return s.at[i] < 0 ? fla_tensor_t{} : gdn_desc(shape, i, static_cast<char*>(s.slab.data_ptr()) + s.at[i]);
  };
  a.q_rstd = piece(GdnSaved::kQr), a.k_rstd = piece(GdnSaved::kKr), a.seg_m = piece(GdnSaved::kSegM);
  const bool normed = s.slab.defined() && s.at[GdnSaved::kQn] >= 0;      // the kernels go on with the normalised rows
  a.q = normed ? piece(GdnSaved::kQn) : desc(q), a.k = normed ? piece(GdnSaved::kKn) : desc(k), a.v = desc(v), a.beta = desc(beta);
  a.gam = piece(GdnSaved::kGam), a.x_inv = piece(GdnSaved::kX), a.s_img = piece(GdnSaved::kS), a.vn_img = piece(GdnSaved::kVn), a.p_img = piece(GdnSaved::kP);
  a.d_o = desc(d_o), a.dht = desc(dht);
  a.dq = desc(dq), a.dk = desc(dk), a.dv = desc(dv), a.dg = desc(dg), a.dbeta = desc(dbeta), a.dh0 = desc(dh0);
  a.cu_seqlens = desc(s.geo.cu), a.chunk_offsets = desc(s.geo.co);
  a.scale = float(scale), a.chunk_size = kChunk, a.max_seqlen = int32_t(s.geo.max_len), a.total_chunks = int32_t(s.geo.chunks);
  two_phase("gdn_chunk_bwd", lib.gdn_chunk_bwd_workspace_size, lib.gdn_chunk_bwd, a, d, true);
  return {dq, dk, dv, dg, dbeta, dh0};
}

// A head-first batch ([B,H,T,D] storage seen as [B,T,H,D]) as one sequence of B*H heads on the same storage; undefined when the
// strides do not allow it.  Every (batch row, head) pair is an independent recurrence, so the kernels run such batches without a copy.
Tensor fold(const Tensor& t) {
  const int64_t B = t.size(0), T = t.size(1), H = t.size(2), D = t.size(3);
  if (t.stride(3) != 1 || t.stride(0) != H * t.stride(2)) return Tensor();
  return t.as_strided({1, T, B * H, D}, {B * t.stride(0), t.stride(1), t.stride(2), 1});
}

std::array<Tensor, 3> fold_plan(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cu) {
  if (cu.defined() || q.dim() != 4 || k.dim() != 4 || v.dim() != 4 || q.size(0) == 1 || (rows_ok(q) && rows_ok(k) && rows_ok(v))) return {};
  std::array<Tensor, 3> f{fold(q), fold(k), fold(v)};
  if (!f[0].defined() || !f[1].defined() || !f[2].defined()) return {};
  return f;
}

struct GdnInputs {      // what the kernels are given: row-major or folded views
  Tensor q, k, v, g, beta, h0;
  bool folded = false;
};
static GdnInputs gdn_inputs(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, const Tensor& h0, const Tensor& cu) {
  GdnInputs in;
  const auto f = fold_plan(q, k, v, cu);
  in.folded = f[0].defined();
  if (in.folded) {      // the gates are re-laid to match (1/128 of the bytes)
    const int64_t B = v.size(0), T = v.size(1), HV = v.size(2);
    in.q = f[0], in.k = f[1], in.v = f[2];
    in.g = g.permute({1, 0, 2}).reshape({1, T, B * HV});
    in.beta = beta.permute({1, 0, 2}).reshape({1, T, B * HV});
    if (h0.defined()) in.h0 = h0.reshape({1, B * HV, h0.size(2), h0.size(3)});
  } else {
    in.q = as_rows(q), in.k = as_rows(k), in.v = as_rows(v), in.g = as_rows(g), in.beta = as_rows(beta), in.h0 = h0;
  }
  return in;
}
static Pair unfold_outputs(const Tensor& o, const Tensor& ht, int64_t B) {
  const int64_t T = o.size(1), HV = o.size(2) / B;
  return {o.view({T, B, HV, o.size(3)}).permute({1, 0, 2, 3}), ht.defined() ? ht.view({B, HV, ht.size(2), ht.size(3)}) : ht};
}

// Saves q, k, v, beta, gam, X and the split per-chunk states / v_new instead of recomputing them.
struct GdnFn : torch::autograd::Function<GdnFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta,
                               const OptTensor& h0_, double scale, bool want_final, const OptTensor& cu_, int64_t out, bool l2norm) {
    const Tensor h0 = value(h0_), cu = value(cu_);
    const GdnInputs in = gdn_inputs(q, k, v, g, beta, h0, cu);
    auto [o, ht, s] = gdn_fwd(in.q, in.k, in.v, in.g, in.beta, scale, in.h0, want_final, cu, true,
                              out < 0 ? std::nullopt : std::optional<at::ScalarType>(at::ScalarType(out)), l2norm, true);
    if (in.folded) std::tie(o, ht) = unfold_outputs(o, ht, q.size(0));
    // with the normalisation in the operator the slab has the rows the backward works on
    ctx->save_for_backward({l2norm ? Tensor() : in.q, l2norm ? Tensor() : in.k, in.v, in.beta, s.slab, s.geo.cu, s.geo.co});
    auto& m = ctx->saved_data;
    std::vector<int64_t> geo{s.geo.N, s.geo.max_len, s.geo.chunks, in.q.size(2)};
    geo.insert(geo.end(), s.at.begin(), s.at.end());
    m["geo"] = std::move(geo);
    m["types"] = std::vector<int64_t>{int64_t(q.scalar_type()), int64_t(k.scalar_type()), int64_t(v.scalar_type()), int64_t(g.scalar_type()),
                                      int64_t(beta.scalar_type())};
    m["fold"] = in.folded ? q.size(0) : int64_t(0);
    m["o"] = o.sizes();
    m["scale"] = scale, m["h0"] = h0.defined();
    ctx->set_materialize_grads(false);
    if (want_final) return {o, ht};
    return {o};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list sv = ctx->get_saved_variables();
    auto& m = ctx->saved_data;
    const std::vector<int64_t> geo = m["geo"].toIntVector(), ty = m["types"].toIntVector();
    GdnSaved s;
    s.slab = sv[4];
    s.geo = Geometry{sv[5], sv[6], geo[0], geo[1], geo[2]};
    s.hk = geo[3];
    std::copy(geo.begin() + 4, geo.end(), s.at.begin());
    const int64_t B = m["fold"].toInt();
    Tensor d_o = grads[0].defined() ? grads[0] : at::zeros(m["o"].toIntVector(), sv[2].options());
    Tensor dht = grads.size() > 1 ? grads[1] : Tensor();
    if (B) {
      const int64_t T = d_o.size(1);
      d_o = d_o.permute({1, 0, 2, 3}).reshape({1, T, -1, d_o.size(3)});      // a view when d_o has the strides of o
      if (dht.defined()) dht = dht.reshape({1, -1, dht.size(2), dht.size(3)});
    }
    // gradients leave the kernels in the dtypes of their inputs
    auto kernel_type = [](int64_t t) { return at::ScalarType(t) == at::kBFloat16 ? at::kBFloat16 : at::kFloat; };
    const GradTypes want{kernel_type(ty[0]), kernel_type(ty[1]), kernel_type(ty[2]), kernel_type(ty[3]), kernel_type(ty[4])};
    auto r = gdn_bwd(sv[0], sv[1], sv[2], sv[3], s, d_o, dht, m["scale"].toDouble(), m["h0"].toBool(), want);
    if (B) {
      for (int i = 0; i < 3; ++i) r[i] = r[i].view({r[i].size(1), B, -1, r[i].size(3)}).permute({1, 0, 2, 3});
      for (int i = 3; i < 5; ++i) r[i] = r[i].view({r[i].size(1), B, -1}).permute({1, 0, 2});
      if (r[5].defined()) r[5] = r[5].view({B, -1, r[5].size(2), r[5].size(3)});
    }
    for (int i = 0; i < 5; ++i) r[i] = r[i].to(at::ScalarType(ty[i]));
    return {r[0], r[1], r[2], r[3], r[4], r[5], Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

Pair gdn(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& g_, const Tensor& beta_, double scale, const Tensor& h0, bool want_final,
         const Tensor& cu, std::optional<at::ScalarType> out, bool l2norm) {
  const char* op = "chunk_gated_delta_rule";
  Tensor q = q_, k = k_, v = v_, g = g_, beta = beta_;
  const bool half = q.scalar_type() == at::kHalf || k.scalar_type() == at::kHalf || v.scalar_type() == at::kHalf;
  std::optional<at::ScalarType> inner = out;
  if (half) {
    // fp16 tensors (the reference takes them, examples/flash_gated_delta_rule.py:1161-1162): the tensor-core products run on
    // bf16 operands, so q, k, v are rounded to bf16 by the library's conversion kernel, fp16 gates become fp32, o is computed
    // in fp32 and converted to fp16 once; the gradients come back through the same conversions
    TORCH_CHECK_TYPE(q.scalar_type() == k.scalar_type() && k.scalar_type() == v.scalar_type(), op, ": q, k, v must share one dtype, got ", q.scalar_type(),
                     ", ", k.scalar_type(), ", ", v.scalar_type());
    q = to_dtype(q, at::kBFloat16, op), k = to_dtype(k, at::kBFloat16, op), v = to_dtype(v, at::kBFloat16, op);
    if (g.scalar_type() == at::kHalf) g = to_dtype(g, at::kFloat, op);
    if (beta.scalar_type() == at::kHalf) beta = to_dtype(beta, at::kFloat, op);
    inner = at::kFloat;
  }
  Pair r;
  if (at::GradMode::is_enabled() && any_requires_grad({q, k, v, g, beta, h0})) {
    variable_list l = GdnFn::apply(q, k, v, g, beta, opt(h0), scale, want_final, opt(cu), inner ? int64_t(*inner) : int64_t(-1), l2norm);
    r = {l[0], l.size() > 1 ? l[1] : Tensor()};
  } else {
    Device(op)(q)(k)(v).get();
    const GdnInputs in = gdn_inputs(q, k, v, g, beta, h0, cu);
    auto [o, ht, s] = gdn_fwd(in.q, in.k, in.v, in.g, in.beta, scale, in.h0, want_final, cu, false, inner, l2norm, true);
    r = in.folded ? unfold_outputs(o, ht, q.size(0)) : Pair{o, ht};
  }
  if (half) r.first = to_dtype(r.first, out.value_or(at::kHalf), op);
  return r;
}

}  // namespace fla_host
