// causal_conv1d: forward, backward (with its autograd node) and the decode update.
#include "runtime.h"
#include <torch/csrc/autograd/custom_function.h>

namespace fla_host {

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// An output with the layout the input has, as torch.empty_like would give it, without its dispatch in the common case.
static Tensor like(const Tensor& x, at::Device d) { return x.is_contiguous() ? empty(x.sizes(), x.scalar_type(), d) : at::empty_like(x); }
static Tensor on_device_i32(const Tensor& t, const Tensor& x) { return t.defined() ? t.to(x.device(), at::kInt) : t; }

Pair conv_fwd(const Tensor& x_, const Tensor& weight, const Tensor& bias, const Tensor& residual, const Tensor& init, bool want_final, bool silu,
              const Tensor& cu_, int64_t head_num) {
  const char* op = "causal_conv1d";
  TORCH_CHECK(x_.dim() == 3, op, ": x must be [B,T,D], got ", x_.sizes());
  const int64_t B = x_.size(0), T = x_.size(1), D = x_.size(2), W = weight.size(1);
  const at::Device d = Device("causal_conv1d_fwd")(x_)(weight)(bias)(residual)(init).get();
  const Tensor x = x_.stride(2) == 1 ? x_ : x_.contiguous();
  const Tensor cu = on_device_i32(cu_, x);
  const int64_t N = cu.defined() ? cu.numel() - 1 : B;
  Tensor y;
  if (head_num > 0) {
    TORCH_CHECK(D % head_num == 0 && (D / head_num) % 8 == 0, op, ": head_num=", head_num, " must divide D=", D, " into heads of a multiple of 8 channels");
    y = empty({B, head_num, T, D / head_num}, x.scalar_type(), d);
  } else {
    y = like(x, d);
  }
  Tensor fin;
  if (want_final) fin = empty({N, D, W - 1}, x.scalar_type(), d);
  fla_causal_conv1d_fwd_args a{};
  a.x = desc(x), a.weight = desc(weight), a.bias = desc(bias), a.residual = desc(residual);
  a.initial_state = desc(init), a.y = desc(y), a.final_state = desc(fin), a.cu_seqlens = desc(cu);
  a.activation_silu = silu;
  two_phase("causal_conv1d_fwd", lib.causal_conv1d_fwd_workspace_size, lib.causal_conv1d_fwd, a, d);
  return {y, fin};
}

std::vector<Tensor> conv_bwd(const Tensor& x_, const Tensor& weight, const Tensor& dy_, const Tensor& bias, const Tensor& init, const Tensor& dht,
                             bool silu, const Tensor& cu_, const Tensor& y_pre, bool want_dh0, at::ScalarType dw_dtype, at::ScalarType db_dtype) {
  const at::Device d = Device("causal_conv1d_bwd")(x_)(weight)(bias)(dy_)(y_pre)(init)(dht).get();
  const int64_t B = x_.size(0), D = x_.size(2), W = weight.size(1);
  const Tensor x = x_.stride(-1) == 1 ? x_ : x_.contiguous();
  Tensor dy = dy_.stride(-1) == 1 && dy_.scalar_type() == x.scalar_type() ? dy_ : dy_.contiguous();
  if (dy.scalar_type() != x.scalar_type()) dy = dy.to(x.scalar_type());
  const Tensor cu = on_device_i32(cu_, x);
  const int64_t N = cu.defined() ? cu.numel() - 1 : B;
  Tensor dx = like(x, d), dw = empty({D, W}, dw_dtype, d), db = empty({D}, db_dtype, d), dh0;
  if (want_dh0) dh0 = at::zeros({N, D, W - 1}, x.options().dtype(at::kFloat));
  fla_causal_conv1d_bwd_args a{};
  a.x = desc(x), a.weight = desc(weight), a.bias = desc(bias), a.dy = desc(dy), a.y_pre = desc(y_pre);
  a.initial_state = desc(init), a.dht = desc(dht);
  a.dx = desc(dx), a.dw = desc(dw), a.db = desc(db), a.dh0 = desc(dh0), a.cu_seqlens = desc(cu);
  a.activation_silu = silu;
  two_phase("causal_conv1d_bwd", lib.causal_conv1d_bwd_workspace_size, lib.causal_conv1d_bwd, a, d);
  return {dx, dw, db, dh0};
}

// Saves the inputs; the backward recomputes the pre-activation.
struct ConvFn : torch::autograd::Function<ConvFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, const OptTensor& bias_, const OptTensor& residual_,
                               const OptTensor& init_, bool want_final, bool silu, const OptTensor& cu_) {
    const Tensor bias = value(bias_), residual = value(residual_), init = value(init_), cu = value(cu_);
    auto [y, fin] = conv_fwd(x, weight, bias, residual, init, want_final, silu, cu, 0);
    ctx->save_for_backward({x, weight, bias, init, cu});
    ctx->saved_data["silu"] = silu;
    ctx->saved_data["residual"] = residual.defined();
    ctx->set_materialize_grads(false);
    if (want_final) return {y, fin};
    return {y};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const Tensor &x = s[0], &weight = s[1], &bias = s[2], &init = s[3];
    const Tensor dy = grads[0].defined() ? grads[0] : at::zeros_like(x);
    Tensor dht;
    if (grads.size() > 1 && grads[1].defined()) dht = grads[1].to(x.scalar_type());
    auto f32_or = [](const Tensor& t) { return t.defined() && t.scalar_type() == at::kBFloat16 ? at::kBFloat16 : at::kFloat; };
    auto g = conv_bwd(x, weight, dy, bias, init, dht, ctx->saved_data["silu"].toBool(), s[4], Tensor(), init.defined(), f32_or(weight), f32_or(bias));
    return {g[0], g[1].to(weight.scalar_type()), bias.defined() ? g[2].to(bias.scalar_type()) : Tensor(),
            ctx->saved_data["residual"].toBool() ? dy : Tensor(), init.defined() ? g[3].to(init.scalar_type()) : Tensor(),
            Tensor(), Tensor(), Tensor()};
  }
};

Pair conv(const Tensor& x, const Tensor& weight, const Tensor& bias, const Tensor& residual, const Tensor& init, bool want_final, bool silu,
          const Tensor& cu) {
  if (!at::GradMode::is_enabled() || !any_requires_grad({x, weight, bias, residual, init}))
    return conv_fwd(x, weight, bias, residual, init, want_final, silu, cu, 0);
  variable_list r = ConvFn::apply(x, weight, opt(bias), opt(residual), opt(init), want_final, silu, opt(cu));
  return {r[0], r.size() > 1 ? r[1] : Tensor()};
}

Tensor conv_update(const Tensor& x, const Tensor& cache, const Tensor& residual, const Tensor& weight, const Tensor& bias, bool silu,
                   const Tensor& cache_indices, const Tensor& accepted, int64_t pad_slot) {
  const char* op = "causal_conv1d_update";
  TORCH_CHECK(!cache.requires_grad(), op, ": cache is updated in place and must not require grad");
  const at::Device d = Device(op)(x)(weight)(bias)(residual)(cache)(cache_indices)(accepted).get();
  Tensor y = like(x, d);
  fla_causal_conv1d_update_args a{};
  auto with_time = [&](const Tensor& t) {      // [N, D] as [N, 1, D]
    fla_tensor_t r = desc(t);
    if (r.ndim == 2) {
      r.ndim = 3;
      r.shape[2] = r.shape[1], r.stride[2] = r.stride[1];
      r.shape[1] = 1, r.stride[1] = r.shape[2] * r.stride[2];
    }
    return r;
  };
  a.x = with_time(x), a.weight = desc(weight), a.bias = desc(bias), a.residual = with_time(residual);
  a.conv_state = desc(cache), a.y = with_time(y), a.cache_indices = desc(cache_indices), a.num_accepted_tokens = desc(accepted);
  a.activation_silu = silu;
  a.pad_slot_id = int32_t(pad_slot);
  two_phase(op, lib.causal_conv1d_update_workspace_size, lib.causal_conv1d_update, a, d);
  cache.unsafeGetTensorImpl()->bump_version();
  return y;
}

}  // namespace fla_host
