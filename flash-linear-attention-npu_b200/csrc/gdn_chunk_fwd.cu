// Chunked gated-delta-rule forward (chunk = 64 tokens, K = V = 128) as two kernels:
//
//  gdn_prep_kernel   (parallel over chunks): gam = chunk-local cumsum(g);
//                    A[i,j] = beta_i exp(gam_i - gam_j) k_i.k_j (j < i);  X = (I + A)^-1
//                    KK^T on tcgen05 (shared by the value heads of a GVA group); the unit lower-triangular inverse by
//                    blocks in fp32 on CUDA cores (tri_inverse.cuh).
//                    Replaces chunk_local_cumsum + chunk_scaled_dot_kkt + solve_tri of the reference
//                    (examples/flash_gated_delta_rule.py:811-838).
//  gdn_scan_fwd_kernel (gdn_scan_fwd.cuh; sequential over chunks, one CTA per (sequence, value head, 128-column block of V)):
//                    v_new = X (beta * (V - exp(gam) * (K S)))
//                    o     = scale (exp(gam) * (Q S) + tril(Q K^T * exp(gam_i - gam_j)) v_new)
//                    S    <- exp(gam_L) S + K^T (exp(gam_L - gam) * v_new)
//                    which is recompute_w_u + chunk_gated_delta_rule_fwd_h + chunk_fwd_o of the reference
//                    (examples/flash_gated_delta_rule.py:840-880) with the WY factors w, u folded away so
//                    that no per-chunk intermediate (A, w, u, h, v_new) round-trips through HBM.
//
// The fp32 state lives in TMEM for the whole sequence.  Tensor-core operands that the result is
// sensitive to (the state copy, beta*(V - ...), v_new, the decayed score tile) are split into a bf16
// "hi" part and a bf16 residual and multiplied in two or three passes; q, k, v enter as the exact
// bf16 inputs.  All matrix products run as tcgen05.mma with M = 128 (unused accumulator rows are
// ignored) so that TMEM lane == accumulator row for every tile.
#include "gdn_common.cuh"
#include "fla_b200_internal.h"
#include "kernel_timer.h"
#include "tri_inverse.cuh"
#include "tensor_map.h"
#include "aux_stream.h"

namespace fla {

struct GdnFwdParams {
  const bf16* q; const bf16* k; const bf16* v;
  bf16* qn; bf16* kn;  // [tokens, HK, K] optional out: q, k rows normalised by the prep kernel; the scan then reads these
  float* q_rstd; float* k_rstd;   // [tokens, HK] their factors
  const void* g; const void* beta;
  float* gam;          // [tokens, HV]      chunk-local cumulative log decay (saved for backward)
  bf16* X;             // [chunks, HV, 2, 8 x 64 x 8]  the chunk's (I + A)^-1 as value + residual strips (saved for backward)
  bf16* p_img;         // [chunks, HV, kPImg]: tril(Q K^T * decay) as value / residual strips, then the chunk's factor record (reused by backward)
  const float* h0;     // [N, HV, K, V] or null
  float* ht;           // [N, HV, K, V] or null
  void* o;             // [tokens, HV, V]
  bf16* s_img;         // [chunks, HV, V/64, 2, 128x64] panel images of the state at chunk start (hi, lo), optional
  bf16* seg_m;         // [segments, HV, 128x128 (value, residual)]  transition matrix of a segment (split chains only)
  float* seg_h;        // [segments, HV, V/128, 128, 128]  its end state from the zero state (segment 0: from the initial one)
  int seg_len;         // chunks per segment
  bf16* vn_img;        // [chunks, HV, V/64, 2, 64x64]  panel images of v_new (hi, lo), optional
  const int32_t* cu_seqlens; const int32_t* chunk_offsets;
  int64_t q_st, q_sh, k_st, k_sh, v_st, v_sh, o_st, o_sh, g_st, beta_st;
  int N, T, HK, HV, g_is_f32, beta_is_f32, o_is_f32;
  int V, nvb;          // value head dim (128 or 256) and its number of 64-column blocks
  float scale;
  int* status;
};

}  // namespace fla
#include "gdn_scan_fwd.cuh"
namespace fla {

// --------------------------------------------------------------------------------------------- prep
// One CTA per (chunk, q/k head).  One M = 128 product [q; k] k^T leaves Q K^T in TMEM lanes 0..63 and K K^T in
// lanes 64..127.  Eight warps: warp w reads lane quadrant w % 4 and the half w / 4 of the 64 columns, so a thread keeps
// half a row (32 values) in registers; per value head of the GVA group the q-side threads emit their half of
// P = tril(Q K^T * e^{gam_i - gam_j}) as split operand panels and the k-side threads their half of A^T, which stays in shared
// memory (where q and k were) and is inverted on the spot, two heads at a time with four warps each: A^T through memory to a kernel
// of its own and back cost 16 KB each way per tile.  (With four warps
// and whole rows per thread the kernel took 0.245 ms at the benchmark shape: it is a chain of latencies, and half the
// work per thread at twice the warps per SM shortens it.)
constexpr int kPrepThreads = 256;
constexpr int kPrepSmem = 2 * kTriTile * 4;      // [q; k] panels (32 KB), then the A^T tiles of two heads
static_assert(kPrepSmem >= 32768, "the panels must fit");
__global__ void __launch_bounds__(kPrepThreads, 4) gdn_prep_kernel(GdnFwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* qk_pan = smem;                        // 2 panels x 128 rows: rows 0..63 q, rows 64..127 k
  __shared__ __align__(16) float gam_s[2][kC];   // gam log2(e): the decays are powers of two of its differences
  __shared__ float wsum_s[4];
  __shared__ uint32_t tmem_base_s;
  __shared__ __align__(8) uint64_t bar;

  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  pdl_trigger();
  pdl_wait();
  const int hk = blockIdx.y;
  const ChunkPos pos = chunk_pos(p.cu_seqlens, p.chunk_offsets, p.N, p.T, 0, blockIdx.x);
  const SeqInfo& sq = pos.sq;
  const int t0 = pos.c * kC;
  const int rows = min(kC, sq.len - t0);
  const int64_t tok0 = int64_t(sq.bos) + t0;
  {
    uint4 val[8];   // all loads in flight before the first one is consumed
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int idx = tid + i * kPrepThreads, r = (idx / 16) & 63, ch = idx % 16;
      const bool isk = idx >= 1024;
      val[i] = make_uint4(0, 0, 0, 0);
      if (r < rows) {
        const bf16* src = isk ? p.k + (tok0 + r) * p.k_st + hk * p.k_sh : p.q + (tok0 + r) * p.q_st + hk * p.q_sh;
        val[i] = *reinterpret_cast<const uint4*>(src + ch * 8);
      }
    }
    // use_qk_l2norm: the sixteen threads that hold a row's pieces normalise it here, where the rows are in registers anyway, and
    // leave it for the scan as well.  As a pass of its own in front (two launches, and two copies when q, k are views of a
    // wider projection) this took 276 us of a 16,384-token prompt's 1,472; in here the kernel grows by what it writes.
    if (p.qn) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int idx = tid + i * kPrepThreads, r = (idx / 16) & 63, ch = idx % 16;
        float x[8], acc = 0.f;
        unpack_bf16x8(val[i], x);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc += x[j] * x[j];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        const float rs = rsqrtf(acc + 1e-6f);
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] *= rs;
        val[i] = pack8(x);
        if (r < rows) {
          const int64_t off = (tok0 + r) * p.HK + hk;
          *reinterpret_cast<uint4*>((idx >= 1024 ? p.kn : p.qn) + off * kK + ch * 8) = val[i];
          if (ch == 0) (idx >= 1024 ? p.k_rstd : p.q_rstd)[off] = rs;
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int idx = tid + i * kPrepThreads, r = ((idx / 16) & 63) + (idx >= 1024 ? 64 : 0), ch = idx % 16;
      *reinterpret_cast<uint4*>(qk_pan + (ch / 8) * 16384 + panel_chunk_off(r, ch % 8)) = val[i];
    }
  }
  if (warp == 0) {
    tmem_alloc(&tmem_base_s, 64);
    tmem_relinquish();
  }
  if (tid == 0) {
    clear_status(p.status, blockIdx.x + hk == 0);
    mbar_init(&bar, 1);
    mbar_init_fence();
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = tmem_base_s;
  if (tid == 0) {
    const Operand a{smem_u32(qk_pan), 16384u, 0};
    const Operand b{smem_u32(qk_pan) + 8192u, 16384u, 0};   // k rows as B (N = 64 tokens)
    mma_tile(tbase, a, b, 128, 64, 8, false);
    mma_commit(&bar);
  }
  const int G = p.HV / p.HK;
  const int quad = warp & 3, half = warp >> 2;
  const int row = quad * 32 + lane;                 // accumulator row == TMEM lane
  const bool kside = row >= 64;
  const int tok = row & 63;
  const int j0 = half * 32;                         // my 32 columns
  // Two value heads at a time.  Their gates are requested a pair ahead (those of the first pair before the product is waited for):
  // warps 0..3 hold g of (head warp / 2, token (warp % 2) * 32 + lane), the k-side threads beta of both heads.
  const int sh = warp >> 1, st = (warp & 1) * 32 + lane;
  auto fetch_g = [&](int h) { return (warp < 4 && h + sh < G && st < rows) ? ld_scalar(p.g, (tok0 + st) * p.g_st + hk * G + h + sh, p.g_is_f32) : 0.f; };
  auto fetch_b = [&](int h) { return (kside && h < G && tok < rows) ? ld_scalar(p.beta, (tok0 + tok) * p.beta_st + hk * G + h, p.beta_is_f32) : 0.f; };
  float g_next = fetch_g(0), b_next[2] = {fetch_b(0), fetch_b(1)};
  const bool ok = __syncthreads_and(mbar_wait(&bar, 0, p.status, FLA_ERR_TIMEOUT));
  tc_fence_after();

  for (int h0 = 0; ok && h0 < G; h0 += 2) {      // (a wait that ran out did so for the whole CTA)
    const int pair = min(2, G - h0);
    float sc[32];   // my half of row `tok` of Q K^T (q side) or K K^T (k side): read again for each pair, the inverse needs the registers
    tmem_ld32(tmem_addr(tbase, quad * 32, j0), sc);
    // chunk-local cumulative sums of g
    float gv = g_next;
    const float bi[2] = {b_next[0], b_next[1]};
    if (h0 + 2 < G) {
      g_next = fetch_g(h0 + 2);
      b_next[0] = fetch_b(h0 + 2);
      b_next[1] = fetch_b(h0 + 3);
    }
    if (warp < 4) {
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, gv, o);
        if (lane >= o) gv += up;
      }
      if (lane == 31) wsum_s[warp] = gv;
    }
    __syncthreads();
    if (warp < 4) {
      if (warp & 1) gv += wsum_s[warp - 1];
      gam_s[sh][st] = gv * kLog2e;
      if (sh < pair && st < rows) p.gam[(tok0 + st) * p.HV + hk * G + h0 + sh] = gv;
    }
    __syncthreads();
    tmem_ld_wait();
    const bool below = j0 <= (quad & 1) * 32 + 31;      // my warp's quarter of the tile reaches below the diagonal
    for (int hh = 0; hh < pair; ++hh) {
      const int64_t cidx = (int64_t(sq.cbase) + pos.c) * p.HV + hk * G + h0 + hh;
      const float* gam = gam_s[hh];
      const float gam_i = gam[tok];
      if (!kside) {
        // my half of the P row as split bf16, in strips of 8 columns ([j / 8][row i][16 bytes], value then residual): the 16
        // bytes a thread stores for a strip lie next to its neighbours' (512 contiguous bytes per warp store), and the scans
        // read the image as an operand with the reduction along j (forward) or along i (reverse) by the descriptor alone
        uint8_t* img = reinterpret_cast<uint8_t*>(p.p_img + cidx * kPImg);
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
          uint4 hi = make_uint4(0, 0, 0, 0), lo = hi;
          if (below) {
            float t[8];
            gather8(gam + j0 + ch * 8, t);
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) {
              const int j = j0 + ch * 8 + jj;
              t[jj] = (j <= tok) ? sc[ch * 8 + jj] * exp2_fast(gam_i - t[jj]) : 0.f;
            }
            split8(t, hi, lo);
          }
          const uint32_t off = uint32_t(half * 4 + ch) * 1024u + uint32_t(tok) * 16u;
          *reinterpret_cast<uint4*>(img + off) = hi;
          *reinterpret_cast<uint4*>(img + 8192 + off) = lo;
        }
      } else {
        const float b = bi[hh];
        if (half == 0) {   // the chunk's per-token factors for the scans, behind the P tile (rows past the end: beta = 0, gam = gam_L)
          ScanFactors* f = reinterpret_cast<ScanFactors*>(reinterpret_cast<uint8_t*>(p.p_img + cidx * kPImg) + kPTileBytes);
          const float eg = exp2_fast(gam_i), gl = gam[rows - 1];
          f->b[tok] = b;
          f->bg[tok] = b * eg;
          f->se[tok] = p.scale * eg;
          f->dk[tok] = exp2_fast(gl - gam_i);
          if (tok == 0) f->dl = exp2_fast(gl);
        }
        // A^T[j][i] = beta_i exp(gam_i - gam_j) (k_i . k_j) for j < i, else 0
        float* at = reinterpret_cast<float*>(smem) + hh * kTriTile;
        if (below) {
#pragma unroll
          for (int ch = 0; ch < 4; ++ch) {
            float t[8];
            gather8(gam + j0 + ch * 8, t);
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) {
              const int j = j0 + ch * 8 + jj;
              at[j * kTriStride + tok] = j < tok ? b * exp2_fast(gam_i - t[jj]) * sc[ch * 8 + jj] : 0.f;
            }
          }
        }
      }
    }
    __syncthreads();
    {      // the tiles are complete: four warps each
      const int grp = tid >> 7, t = tid & 127;
      if (grp < pair) {
        float* tile = reinterpret_cast<float*>(smem) + grp * kTriTile;
        tri_invert<128>(tile, t, 1 + grp);
        tri_store_strips<128>(tile, reinterpret_cast<uint8_t*>(p.X + ((int64_t(sq.cbase) + pos.c) * p.HV + hk * G + h0 + grp) * 8192), rows, t);
      }
    }
    if (h0 + 2 < G) __syncthreads();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tbase, 64);
}

}  // namespace fla

using namespace fla;

static int geometry(const fla_gdn_chunk_fwd_args* a, int64_t* total_chunks, int* N, int* max_len) {
  const int64_t B = a->q.shape[0], T = a->q.shape[1];
  *N = int(B);
  *total_chunks = B * ((T + kC - 1) / kC);
  *max_len = int(T);
  if (a->cu_seqlens.data) {
    if (B != 1 || a->cu_seqlens.dtype != FLA_I32 || a->cu_seqlens.ndim != 1 || a->cu_seqlens.shape[0] < 2) return FLA_ERR_SHAPE;
    *N = int(a->cu_seqlens.shape[0] - 1);
    if (!a->chunk_offsets.data || a->chunk_offsets.dtype != FLA_I32 || a->chunk_offsets.shape[0] != *N + 1) return FLA_ERR_SHAPE;
    if (a->max_seqlen <= 0 || a->max_seqlen > T || a->total_chunks <= 0) return FLA_ERR_VALUE;
    *max_len = a->max_seqlen;
    *total_chunks = a->total_chunks;
  }
  return FLA_OK;
}
static SegPlan plan_of(const fla_gdn_chunk_fwd_args* a, int64_t total_chunks, int N, int max_len) {
  SegPlan whole;
  whole.count = N;
  if (a->s_img.data && !a->seg_m.data) return whole;      // the backward has to find the same segments' M
  return scan_plan(N, total_chunks, max_len, a->cu_seqlens.data != nullptr, a->v.shape[2], a->v.shape[3]);
}

// Size of the seg_m buffer a training forward keeps for its backward (0: the chains of this shape are not split).
extern "C" FLA_API int fla_b200_gdn_chunk_segments_size(const fla_gdn_chunk_fwd_args* a, uint64_t* bytes) {
  if (!a || !bytes) return FLA_ERR_NULL;
  if (!a->q.data || a->q.ndim != 4 || !a->v.data || a->v.ndim != 4) return FLA_ERR_SHAPE;
  int64_t total_chunks; int N, max_len;
  if (int st = geometry(a, &total_chunks, &N, &max_len)) return st;
  const SegPlan plan = scan_plan(N, total_chunks, max_len, a->cu_seqlens.data != nullptr, a->v.shape[2], a->v.shape[3]);
  *bytes = plan.split ? uint64_t(plan.count) * a->v.shape[2] * kSegMBytes : 0;
  return FLA_OK;
}

static int check_token_tensor(const fla_tensor_t& t, int64_t heads, int64_t dim, int dtype_a, int dtype_b) {
  // [B, T, H, D] with D contiguous, rows 16-byte aligned, and batch rows laid out back to back
  if (!t.data) return FLA_ERR_NULL;
  if (t.ndim != 4 || t.shape[2] != heads || t.shape[3] != dim) return FLA_ERR_SHAPE;
  if (t.dtype != dtype_a && t.dtype != dtype_b) return FLA_ERR_DTYPE;
  const int64_t esz = t.dtype == FLA_F32 ? 4 : 2;
  if (t.stride[3] != 1 || (t.stride[2] * esz) % 16 || (t.stride[1] * esz) % 16 || !aligned16(t.data)) return FLA_ERR_LAYOUT;
  if (t.shape[0] > 1 && t.stride[0] != t.shape[1] * t.stride[1]) return FLA_ERR_LAYOUT;
  return FLA_OK;
}
static int check_gate_tensor(const fla_tensor_t& t, int64_t B, int64_t T, int64_t heads) {
  if (!t.data) return FLA_ERR_NULL;
  if (t.ndim != 3 || t.shape[0] != B || t.shape[1] != T || t.shape[2] != heads) return FLA_ERR_SHAPE;
  if (t.dtype != FLA_F32 && t.dtype != FLA_BF16) return FLA_ERR_DTYPE;
  if (t.stride[2] != 1 || (B > 1 && t.stride[0] != T * t.stride[1])) return FLA_ERR_LAYOUT;
  return FLA_OK;
}

static uint64_t workspace_bytes_of(const fla_gdn_chunk_fwd_args* a, int64_t chunks, const SegPlan& plan) {
  const uint64_t HV = a->v.shape[2];
  uint64_t b = 256 + uint64_t(chunks) * HV * (a->p_img.data ? 0 : kPImgBytes);
  if (plan.split) b += uint64_t(plan.count) * HV * ((a->seg_m.data ? 0 : kSegMBytes) + kSegHBytes * (a->v.shape[3] / 128));
  return b;
}
extern "C" FLA_API int fla_b200_gdn_chunk_fwd_workspace_size(const fla_gdn_chunk_fwd_args* a, uint64_t* bytes) {
  if (!a || !bytes) return FLA_ERR_NULL;
  if (!a->q.data || a->q.ndim != 4 || !a->v.data || a->v.ndim != 4) return FLA_ERR_SHAPE;
  int64_t chunks; int N, max_len;
  if (int st = geometry(a, &chunks, &N, &max_len)) return st;
  if (chunks <= 0) return FLA_ERR_VALUE;
  // status block + P panels (unless the caller keeps them for the backward) + M and H of the segments of split chains
  *bytes = workspace_bytes_of(a, chunks, plan_of(a, chunks, N, max_len));
  return FLA_OK;
}

extern "C" FLA_API int fla_b200_gdn_chunk_fwd(const fla_gdn_chunk_fwd_args* a, void* workspace, uint64_t workspace_bytes,
                                              void* stream) {
  if (!a) return FLA_ERR_NULL;
  if (!workspace || workspace_bytes < 256 || !aligned16(workspace)) return FLA_ERR_WORKSPACE;
  const fla_tensor_t &q = a->q, &k = a->k, &v = a->v, &o = a->o;
  if (!q.data || !k.data || !v.data || !o.data) return FLA_ERR_NULL;
  if (q.ndim != 4 || v.ndim != 4) return FLA_ERR_SHAPE;
  const int64_t B = q.shape[0], T = q.shape[1], HK = q.shape[2], HV = v.shape[2];
  if (B <= 0 || T <= 0 || HK <= 0 || HV <= 0 || HV % HK || v.shape[0] != B || v.shape[1] != T) return FLA_ERR_SHAPE;
  int st;
  if ((st = check_token_tensor(q, HK, kK, FLA_BF16, FLA_BF16))) return st;
  if ((st = check_token_tensor(k, HK, kK, FLA_BF16, FLA_BF16))) return st;
  const int64_t V = v.shape[3];
  if (V != kV && V != 2 * kV) return FLA_ERR_SHAPE;
  if ((st = check_token_tensor(v, HV, V, FLA_BF16, FLA_BF16))) return st;
  if ((st = check_token_tensor(o, HV, V, FLA_BF16, FLA_F32))) return st;
  if (k.shape[0] != B || k.shape[1] != T || o.shape[0] != B || o.shape[1] != T) return FLA_ERR_SHAPE;
  if ((st = check_gate_tensor(a->g, B, T, HV))) return st;
  if ((st = check_gate_tensor(a->beta, B, T, HV))) return st;
  if (a->chunk_size != kC) return FLA_ERR_VALUE;
  if (!(a->scale == a->scale)) return FLA_ERR_VALUE;

  int N, max_len;
  int64_t total_chunks;
  if ((st = geometry(a, &total_chunks, &N, &max_len))) return st;
  const SegPlan plan = plan_of(a, total_chunks, N, max_len);
  const fla_tensor_t &gam = a->gam, &X = a->x_inv;
  if (!gam.data || !X.data) return FLA_ERR_NULL;
  if (gam.dtype != FLA_F32 || gam.ndim != 3 || gam.shape[0] != B || gam.shape[1] != T || gam.shape[2] != HV ||
      gam.stride[2] != 1 || gam.stride[1] != HV || (B > 1 && gam.stride[0] != T * HV))
    return FLA_ERR_SHAPE;
  if (X.dtype != FLA_BF16 || X.ndim != 1 || X.shape[0] != total_chunks * HV * 8192 || !aligned16(X.data))
    return FLA_ERR_SHAPE;
  for (const fla_tensor_t* s : {&a->initial_state, &a->final_state}) {
    if (!s->data) continue;
    if (s->dtype != FLA_F32) return FLA_ERR_DTYPE;
    if (s->ndim != 4 || s->shape[0] != N || s->shape[1] != HV || s->shape[2] != kK || s->shape[3] != V) return FLA_ERR_SHAPE;
    if (s->stride[3] != 1 || s->stride[2] != V || s->stride[1] != kK * V || s->stride[0] != HV * kK * V || !aligned16(s->data))
      return FLA_ERR_LAYOUT;
  }
  GdnFwdParams p{};
  p.q = static_cast<const bf16*>(q.data); p.k = static_cast<const bf16*>(k.data); p.v = static_cast<const bf16*>(v.data);
  p.g = a->g.data; p.beta = a->beta.data;
  p.gam = static_cast<float*>(gam.data); p.X = static_cast<bf16*>(X.data);
  p.h0 = static_cast<const float*>(a->initial_state.data); p.ht = static_cast<float*>(a->final_state.data);
  p.o = o.data;
  if (a->s_img.data || a->vn_img.data) {
    const fla_tensor_t &si = a->s_img, &vi = a->vn_img;
    if (!si.data || !vi.data) return FLA_ERR_NULL;
    if (si.dtype != FLA_BF16 || si.ndim != 1 || si.shape[0] != total_chunks * HV * (V / kBV) * 16384 || !aligned16(si.data)) return FLA_ERR_SHAPE;
    if (vi.dtype != FLA_BF16 || vi.ndim != 1 || vi.shape[0] != total_chunks * HV * (V / kBV) * 8192 || !aligned16(vi.data)) return FLA_ERR_SHAPE;
    p.s_img = static_cast<bf16*>(si.data);
    p.vn_img = static_cast<bf16*>(vi.data);
  }
  p.cu_seqlens = static_cast<const int32_t*>(a->cu_seqlens.data);
  p.chunk_offsets = static_cast<const int32_t*>(a->chunk_offsets.data);
  p.q_st = q.stride[1]; p.q_sh = q.stride[2]; p.k_st = k.stride[1]; p.k_sh = k.stride[2];
  p.v_st = v.stride[1]; p.v_sh = v.stride[2]; p.o_st = o.stride[1]; p.o_sh = o.stride[2];
  p.g_st = a->g.stride[1]; p.beta_st = a->beta.stride[1];
  p.N = N; p.T = int(T); p.HK = int(HK); p.HV = int(HV); p.V = int(V); p.nvb = int(V / kBV);
  p.g_is_f32 = a->g.dtype == FLA_F32; p.beta_is_f32 = a->beta.dtype == FLA_F32; p.o_is_f32 = o.dtype == FLA_F32;
  p.scale = a->scale;
  p.status = static_cast<int*>(workspace);
  {
    const uint64_t per = uint64_t(total_chunks) * HV;
    if (workspace_bytes < workspace_bytes_of(a, total_chunks, plan)) return FLA_ERR_WORKSPACE;
    if (a->p_img.data) {
      const fla_tensor_t& pi = a->p_img;
      if (pi.dtype != FLA_BF16 || pi.ndim != 1 || pi.shape[0] != int64_t(per) * kPImg || !aligned16(pi.data)) return FLA_ERR_SHAPE;
      p.p_img = static_cast<bf16*>(pi.data);
    } else {
      p.p_img = reinterpret_cast<bf16*>(static_cast<uint8_t*>(workspace) + 256);
    }
    p.seg_len = plan.len;
    if (plan.split) {
      uint8_t* ws = static_cast<uint8_t*>(workspace) + 256 + (a->p_img.data ? 0 : per * kPImgBytes);
      if (a->seg_m.data) {
        if (a->seg_m.dtype != FLA_BF16 || a->seg_m.ndim != 1 || uint64_t(a->seg_m.shape[0]) * 2 < uint64_t(plan.count) * HV * kSegMBytes || !aligned16(a->seg_m.data))
          return FLA_ERR_SHAPE;
        p.seg_m = static_cast<bf16*>(a->seg_m.data);
      } else {
        p.seg_m = reinterpret_cast<bf16*>(ws);
        ws += uint64_t(plan.count) * HV * kSegMBytes;
      }
      p.seg_h = reinterpret_cast<float*>(ws);
    }
  }

  if (a->q_norm.data || a->k_norm.data || a->q_rstd.data || a->k_rstd.data) {
    for (const fla_tensor_t* t : {&a->q_norm, &a->k_norm, &a->q_rstd, &a->k_rstd}) {
      const bool row = t == &a->q_norm || t == &a->k_norm;
      if (!t->data) return FLA_ERR_NULL;
      if (t->dtype != (row ? FLA_BF16 : FLA_F32)) return FLA_ERR_DTYPE;
      if (t->ndim != (row ? 4 : 3) || t->shape[0] != B || t->shape[1] != T || t->shape[2] != HK || (row && t->shape[3] != kK)) return FLA_ERR_SHAPE;
      const int64_t w = row ? kK : 1;
      if ((row && (t->stride[3] != 1 || !aligned16(t->data))) || t->stride[2] != w || t->stride[1] != HK * w || (B > 1 && t->stride[0] != T * HK * w))
        return FLA_ERR_LAYOUT;
    }
    p.qn = static_cast<bf16*>(a->q_norm.data); p.kn = static_cast<bf16*>(a->k_norm.data);
    p.q_rstd = static_cast<float*>(a->q_rstd.data); p.k_rstd = static_cast<float*>(a->k_rstd.data);
  }

  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  const int prep_smem = kPrepSmem + 1024;
  static std::atomic<bool> attr_done_dev[64] = {};   // per device ordinal; setting the attributes twice is harmless
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return FLA_ERR_CUDA;
  std::atomic<bool>& attr_done = attr_done_dev[dev];
  if (!attr_done) {
    if (cudaFuncSetAttribute(gdn_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, prep_smem) != cudaSuccess) return FLA_ERR_CUDA;
    for (auto* scan : {gdn_scan_fwd_kernel<kScanInfer, false>, gdn_scan_fwd_kernel<kScanSave, false>, gdn_scan_fwd_kernel<kScanInfer, true>,
                       gdn_scan_fwd_kernel<kScanSave, true>, gdn_scan_fwd_kernel<kScanState, true>})
      if (cudaFuncSetAttribute(scan, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kScanFwdSmem) + 1024) != cudaSuccess) return FLA_ERR_CUDA;
    attr_done = true;
  }
  {
    KernelTimer kt("gdn_prep", cs);
    if (launch_pdl(gdn_prep_kernel, dim3(unsigned(total_chunks), unsigned(HK)), kPrepThreads, prep_smem, cs, p) != cudaSuccess) return FLA_ERR_CUDA;
  }
  CUtensorMap tm_q, tm_k;
  const uint64_t nst = uint64_t(HK) * kK;   // the normalised rows are dense
  if (p.qn ? (make_row_tile_map(&tm_q, p.qn, kK, uint64_t(HK), uint64_t(B * T), kK, nst) ||
              make_row_tile_map(&tm_k, p.kn, kK, uint64_t(HK), uint64_t(B * T), kK, nst))
           : (make_row_tile_map(&tm_q, p.q, kK, uint64_t(HK), uint64_t(B * T), uint64_t(p.q_sh), uint64_t(p.q_st)) ||
              make_row_tile_map(&tm_k, p.k, kK, uint64_t(HK), uint64_t(B * T), uint64_t(p.k_sh), uint64_t(p.k_st))))
    return FLA_ERR_CUDA;
  CUtensorMap tm_v;
  if (make_row_tile_map(&tm_v, p.v, uint64_t(V), uint64_t(HV), uint64_t(B * T), uint64_t(p.v_sh), uint64_t(p.v_st))) return FLA_ERR_CUDA;
  {
    KernelTimer kt("gdn_fwd", cs);
    const unsigned heads = unsigned(HV * (V / 128));
    if (plan.split && launch_pdl(gdn_scan_fwd_kernel<kScanState, true>, dim3(heads, unsigned(plan.count), 2), kFwdThreads, kScanFwdSmem + 1024, cs, p, tm_q,
                                 tm_k, tm_v) != cudaSuccess)
      return FLA_ERR_CUDA;
    auto* scan = plan.split ? (p.s_img ? gdn_scan_fwd_kernel<kScanSave, true> : gdn_scan_fwd_kernel<kScanInfer, true>)
                            : (p.s_img ? gdn_scan_fwd_kernel<kScanSave, false> : gdn_scan_fwd_kernel<kScanInfer, false>);
    return cuda_status(launch_pdl(scan, dim3(heads, unsigned(plan.count)), kFwdThreads, kScanFwdSmem + 1024, cs, p, tm_q, tm_k, tm_v));
  }
}


