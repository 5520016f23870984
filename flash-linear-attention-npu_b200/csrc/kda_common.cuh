// Parameter block and image sizes shared by the KDA chunk forward and backward translation units.
#pragma once
#include "gdn_common.cuh"
#include "fla_b200_internal.h"

namespace fla {

struct KdaParams {
  const bf16* q; const bf16* k; const bf16* v;
  const void* g; const void* beta;
  float* q_rstd; float* k_rstd;   // [tokens, HK] optional out: when given, the prep kernel normalises the rows of q and k first
  const float* a_log; const float* dt_bias;   // optional gate parameters: [HV], [HV, K]
  float* gk_out;        // [tokens, HV, K] cumulative gate (optional)
  bf16* qk_img;         // [chunks, HV, {hi, lo}, 2 panels x 128 rows]  rows 0-63 Qp, rows 64-127 Kp
  bf16* kn_img;         // [chunks, HV, {hi, lo}, 2 panels x 64 rows]
  bf16* p_img;          // [chunks, HV, {hi, lo}, 64 x 64]   tril(Qp Kn^T)
  bf16* x_img;          // [chunks, HV, {hi, lo}, 64 x 64]   (I + Akk)^-1 
  float* vec;           // [chunks, HV, 4, K]  e^a, e^{gk_L - a}, a, beta of the chunk's tokens
  bf16* s_img;          // optional out for the backward: [chunks, HV, V/64, {hi, lo}, 16 strips of 8 key dims, 64 channels]  Sa = diag(e^a) S at chunk start
  bf16* vn_img;         // optional out for the backward: [chunks, HV, V/64, {hi, lo}, 8 strips of 8 tokens, 64 channels]   v_new
  bf16* seg_m;          // split chains: [segments, HV, 128x128 (value, residual)]  transition matrix of a segment
  float* seg_h;         // split chains: [segments, HV, V/128, 128, 128]  its end state
  int seg_len;          // chunks per segment
  const float* h0; float* ht;
  void* o;              // may be null when only the saved images are wanted
  const int32_t* cu_seqlens; const int32_t* chunk_offsets;
  int64_t q_st, q_sh, k_st, k_sh, v_st, v_sh, o_st, o_sh, g_st, g_sh, beta_st;
  int64_t total_tokens;   // rows of the flat [tokens, heads, dim] views
  int N, T, HK, HV, g_is_f32, beta_is_f32, o_is_f32, gate_mode;
  int V, nvb;           // value head dim (128 or 256) and its number of 64-column blocks
  float scale, lower_bound;
  int* status;
};

constexpr int64_t kKdaQkImg = 32768, kKdaKnImg = 16384, kKdaPImg = 8192, kKdaXImg = 8192;  // bf16 elements, hi + lo
constexpr int64_t kKdaSImg = 16384, kKdaVnImg = 8192;   // per 64-column block of V
constexpr int kKdaVecs = 4;
// The per-chunk record of the prep kernel: factors per key dim and beta per token.
struct __align__(16) KdaFactors {
  float ea[kK];      // e^a
  float el[kK];      // e^{gk_L - a}
  float a[kK];       // the anchor
  float b[kK];       // beta of the chunk's 64 tokens (zero past the end), then unused
};
static_assert(sizeof(KdaFactors) == kKdaVecs * kK * 4, "record size");

// Workspace layout of the forward (offsets of qk_img, kn_img, p_img, x_img, vec); returns the total size.
uint64_t kda_ws_layout(int64_t total_chunks, int64_t HV, uint64_t off[5]);
// Layout of the buffer a training forward leaves for the backward: the forward workspace (operand images), gk, the
// Sa images, the v_new images and the segments' M; returns the total size.
uint64_t kda_saved_layout(int64_t total_chunks, int64_t HV, int64_t nvb, int64_t tokens, int64_t segments, uint64_t off[5]);
// q_rstd, k_rstd of an argument block: both absent, or both dense [B, T, HK] f32; an FLA_ERR_* status otherwise.
int kda_check_rstd(const fla_tensor_t& q, const fla_tensor_t& k, int64_t B, int64_t T, int64_t HK);
// prep -> forward scan on `stream`; 0 or an FLA_ERR_* status.
int kda_launch_forward(const KdaParams& p, int64_t total_chunks, int64_t segments, cudaStream_t stream);

}  // namespace fla
