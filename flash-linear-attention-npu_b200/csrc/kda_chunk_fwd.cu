// Chunked Kimi-Delta-Attention forward (per-channel log gate g[t, h, :], chunk = 64, K = V = 128).
//
//   gk = chunk-local cumsum(gate(g));   with a per-channel anchor a = gk at the middle token of the chunk:
//   Qp = Q * e^{gk - a}   Kp = K * e^{gk - a}   Kn = K * e^{a - gk}        (all finite for any realistic decay)
//   Aqk = tril(Qp Kn^T)   Akk = strict_tril(beta_i Kp Kn^T)   X = (I + Akk)^-1
//   per chunk, Sa = diag(e^a) S:   v_new = X (beta * (V - Kp Sa))
//                                  o     = scale (Qp Sa + Aqk v_new)
//                                  S    <- diag(e^{gk_L - a}) (Sa + Kn^T v_new)
// which equals the reference's chunk_kda_fwd stages (gate cumsum -> Prepare -> Post-WU -> FwdH -> Finalize,
// fla/ops/ascendc/kda/chunk_kda_fwd/docs/design.md:11-78; golden tests/atk/chunk_kda_fwd/executor_chunk_kda_fwd.py:402-530)
// with w, u folded away.  The decay sits inside the K reduction, so the scaled operands cannot be the exact
// bf16 inputs: kda_prep_kernel (parallel over chunks) builds them once as bf16 hi + residual operand panels,
// computes both score tiles on tcgen05 and the inverse on CUDA cores, and stores everything as ready-to-load
// panel images; kda_scan_fwd_kernel (kda_scan_fwd.cuh; sequential over chunks, fp32 state in TMEM) only bulk-loads them.
#include <algorithm>
#include "gdn_common.cuh"
#include "fla_b200_internal.h"
#include "aux_stream.h"
#include "kernel_timer.h"
#include "tri_inverse.cuh"
#include "kda_common.cuh"
#include "tensor_map.h"
#include "kda_scan_fwd.cuh"

namespace fla {

// --------------------------------------------------------------------------------------------- prep
constexpr uint32_t pOffQKH = 0, pOffQKL = 32768, pOffKNH = 65536, pOffKNL = 81920;
// Once the panels are free: the image of P where Qp was, A^T (inverted in place) and the image of X where Kn was, and the next tile's rows
// of q and k where the residuals of Qp and Kp were.
constexpr uint32_t kStageP = pOffQKH, kStageA = pOffKNH, kStageX = pOffKNH + kTriTile * 4;
constexpr uint32_t kKdaPrepSmem = kStageX + 16384;
static_assert(kStageX % 1024 == 0 && kKdaPrepSmem >= pOffKNL + 16384, "panel alignment");

__device__ __forceinline__ float kda_gate(float g, int mode, float eig, float bias, float lower_bound) {
  if (mode == 0) return g;
  const float raw = g + bias;
  if (mode == 1) {  // -exp(A_log) * softplus(g + dt_bias)
    // softplus(x) = max(x, 0) + log1p(e), e = exp(-|x|);  log1p(e) = 2 atanh(s), s = e / (2 + e) <= 1/3, by its series (what is
    // left out is below 2e-8 of it)
    const float e = __expf(-fabsf(raw)), s = __fdividef(e, 2.f + e), z = s * s;
    float a = 1.f / 13;
    a = a * z + 1.f / 11; a = a * z + 1.f / 9; a = a * z + 1.f / 7; a = a * z + 1.f / 5; a = a * z + 1.f / 3; a = a * z + 1.f;
    return -eig * (fmaxf(raw, 0.f) + 2.f * s * a);
  }
  return __fdividef(lower_bound, 1.f + __expf(-eig * raw));  // lower_bound * sigmoid(exp(A_log) (g + dt_bias))
}

// Two CTAs of sixteen warps per SM (what 97 KB of operand panels leave room for), each working through every 2 x #SM-th tile.  Thread
// layout of the elementwise phases: 16 channel groups (8 channels each) x 32 token pairs.  The raw q and k rows arrive as TMA tiles in the
// residual panels, where each thread later overwrites exactly the 16-byte pieces it read; those of the next tile are requested as
// soon as the images have left, and its gates are brought into L2, so that no tile starts with a round trip to HBM.  After the score product the
// warps part: eight write P, eight invert.  What bounds it: instruction issue in the elementwise phases (45 % over all) and the barriers
// between the phases.  8,192 tokens of 32 heads with gate and normalisation: 318 us with eight warps per CTA and one tile
// per CTA, 288 with sixteen warps, 274 now.
constexpr int kKdaPrepThreads = 512, kLeaderK = 64;      // kLeaderK: the thread that issues for the k-side warps (0 for the q-side)
__global__ void __launch_bounds__(kKdaPrepThreads, 2) kda_prep_kernel(KdaParams p, unsigned tiles, const __grid_constant__ CUtensorMap tm_q,
                                                                      const __grid_constant__ CUtensorMap tm_k) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(16) float tot_s[16][kK];      // gate sum of each warp's four tokens, per channel
  __shared__ __align__(16) float anchor_s[kK], last_s[kK];
  __shared__ uint32_t tmem_base_s;
  __shared__ __align__(8) uint64_t bar, qk_bar;

  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  pdl_trigger();
  pdl_wait();
  const int cg = tid & 15, r0 = cg * 8, tb = (tid >> 4) * 2;      // my channels and my first token
  const int quad = warp & 3, j0 = (warp >> 2) * 16, row = quad * 32 + lane, tok = row & 63;      // my 16 score columns of my row
  const int gva = p.HV / p.HK;
  const uint32_t sb = smem_u32(smem);

  // a tile is a (chunk, head); heads fastest, so that the CTAs of one moment read neighbouring pieces of the same token rows
  struct Tile { int hv, tok0, rows; };
  auto tile_at = [&](unsigned tile) {
    const unsigned chunk = tile / unsigned(p.HV);
    const ChunkPos pos = chunk_pos(p.cu_seqlens, p.chunk_offsets, p.N, p.T, 0, int(chunk));
    return Tile{int(tile - chunk * unsigned(p.HV)), pos.sq.bos + pos.c * kC, min(kC, pos.sq.len - pos.c * kC)};
  };
  auto load_qk = [&](const Tile& t) {      // one thread
    const int hk = t.hv / gva;
    mbar_arrive_expect_tx(&qk_bar, 4 * 8192);
    tma_load_tile(sb + pOffQKL, &tm_q, 0, hk, t.tok0, &qk_bar);                  // q rows -> rows 0-63 of the residual panels
    tma_load_tile(sb + pOffQKL + 16384, &tm_q, 64, hk, t.tok0, &qk_bar);
    tma_load_tile(sb + pOffQKL + 8192, &tm_k, 0, hk, t.tok0, &qk_bar);           // k rows -> rows 64-127
    tma_load_tile(sb + pOffQKL + 16384 + 8192, &tm_k, 64, hk, t.tok0, &qk_bar);
  };

  if (warp == 0) {
    tmem_alloc(&tmem_base_s, 64);
    tmem_relinquish();
  }
  Tile cur = tile_at(blockIdx.x);
  if (tid == 0) {
    clear_status(p.status, blockIdx.x == 0);
    mbar_init(&bar, 1);
    mbar_init(&qk_bar, 1);
    mbar_init_fence();
    load_qk(cur);
  }
  uint32_t parity = 0;
  for (unsigned tile = blockIdx.x; tile < tiles; tile += gridDim.x, parity ^= 1) {
  const int hv = cur.hv, rows = cur.rows;
  const int64_t tok0 = cur.tok0, cidx = tile;
  // 1. activated gates of my 2 tokens x 8 channels (zero past the sequence end), summed over the warp's tokens before them
  float gk[2][8];
  {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
#pragma unroll
      for (int j = 0; j < 8; ++j) gk[i][j] = 0.f;
      if (tb + i < rows) {
        const int64_t off = (tok0 + tb + i) * p.g_st + hv * p.g_sh + r0;
        if (p.g_is_f32) gather8(static_cast<const float*>(p.g) + off, gk[i]);
        else unpack_bf16x8(*reinterpret_cast<const uint4*>(static_cast<const bf16*>(p.g) + off), gk[i]);
      }
    }
    if (p.gate_mode) {
      const float eig = p.a_log ? __expf(p.a_log[hv]) : 1.f;
      float bias[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) bias[j] = 0.f;
      if (p.dt_bias) gather8(p.dt_bias + hv * kK + r0, bias);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) gk[i][j] = tb + i < rows ? kda_gate(gk[i][j], p.gate_mode, eig, bias[j], p.lower_bound) : 0.f;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      gk[1][j] += gk[0][j];
      const float below = __shfl_up_sync(0xffffffffu, gk[1][j], 16);
      if (lane >= 16) {
        gk[0][j] += below;
        gk[1][j] += below;
      }
    }
    if (lane >= 16) {
      *reinterpret_cast<float4*>(&tot_s[warp][r0]) = make_float4(gk[1][0], gk[1][1], gk[1][2], gk[1][3]);
      *reinterpret_cast<float4*>(&tot_s[warp][r0 + 4]) = make_float4(gk[1][4], gk[1][5], gk[1][6], gk[1][7]);
    }
  }
  if (tid == 0 || tid == kLeaderK) bulk_wait_read();     // the previous tile's P and X have left shared memory
  __syncthreads();
  // 2. add the totals of the earlier warps; publish the anchor row (middle token) and the last valid row
  {
    float off[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) off[j] = 0.f;
    for (int w = 0; w < warp; ++w) {
      float t[8];
      gather8(&tot_s[w][r0], t);
#pragma unroll
      for (int j = 0; j < 8; ++j) off[j] += t[j];
    }
    const int ta = min(kC / 2 - 1, rows - 1), tl = rows - 1;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
#pragma unroll
      for (int j = 0; j < 8; ++j) gk[i][j] += off[j];
      if (tb + i == ta) {
#pragma unroll
        for (int j = 0; j < 8; ++j) anchor_s[r0 + j] = gk[i][j];
      }
      if (tb + i == tl) {
#pragma unroll
        for (int j = 0; j < 8; ++j) last_s[r0 + j] = gk[i][j];
      }
    }
  }
  __syncthreads();
  if (tid < kK) {
    const float a = anchor_s[tid];
    p.vec[cidx * kKdaVecs * kK + tid] = __expf(a);
    p.vec[cidx * kKdaVecs * kK + kK + tid] = __expf(last_s[tid] - a);
    p.vec[cidx * kKdaVecs * kK + 2 * kK + tid] = a;
  } else if (tid < 2 * kK) {
    const int t = tid - kK;
    p.vec[cidx * kKdaVecs * kK + 3 * kK + t] = t < rows ? ld_scalar(p.beta, (tok0 + t) * p.beta_st + hv, p.beta_is_f32) : 0.f;
  }
  // 3. scaled operands as split bf16 panels
  {
    const uint32_t pan = (cg / 8) * 16384, pan64 = (cg / 8) * 8192;
    const bool landed = mbar_wait(&qk_bar, parity, p.status, FLA_ERR_TIMEOUT);
    if (p.gk_out) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (tb + i < rows) {
          float* dst = p.gk_out + ((tok0 + tb + i) * p.HV + hv) * kK + r0;
          *reinterpret_cast<float4*>(dst) = make_float4(gk[i][0], gk[i][1], gk[i][2], gk[i][3]);
          *reinterpret_cast<float4*>(dst + 4) = make_float4(gk[i][4], gk[i][5], gk[i][6], gk[i][7]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = tb + i;
      const uint32_t o1 = panel_chunk_off(t, cg % 8), o2 = panel_chunk_off(64 + t, cg % 8);
      float qv[8], kv[8];
      uint4 qraw = make_uint4(0, 0, 0, 0), kraw = qraw;
      if (t < rows && landed) {   // rows past the end of the sequence hold foreign tokens in the tile: use zeros
        qraw = *reinterpret_cast<const uint4*>(smem + pOffQKL + pan + o1);
        kraw = *reinterpret_cast<const uint4*>(smem + pOffQKL + pan + o2);
      }
      unpack_bf16x8(qraw, qv);
      unpack_bf16x8(kraw, kv);
      // use_qk_l2norm: x * rsqrt(sum x^2 + 1e-6) rounded to bf16; the sixteen threads of a token hold its row.  As two passes in
      // front of this kernel it took 115 us of an 8,192-token prompt's 946.
      if (p.q_rstd) {
        float sq_q = 0.f, sq_k = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) { sq_q += qv[j] * qv[j]; sq_k += kv[j] * kv[j]; }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
          sq_q += __shfl_xor_sync(0xffffffffu, sq_q, o);
          sq_k += __shfl_xor_sync(0xffffffffu, sq_k, o);
        }
        const float rq = rsqrtf(sq_q + 1e-6f), rk = rsqrtf(sq_k + 1e-6f);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          qv[j] *= rq;
          kv[j] *= rk;
        }
        unpack_bf16x8(pack8(qv), qv);
        unpack_bf16x8(pack8(kv), kv);
        if (cg == 0 && t < rows && hv % gva == 0) {
          p.q_rstd[(tok0 + t) * p.HK + hv / gva] = rq;
          p.k_rstd[(tok0 + t) * p.HK + hv / gva] = rk;
        }
      }
      float an[8], kn[8];
      gather8(&anchor_s[r0], an);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float d = (gk[i][j] - an[j]) * kLog2e;
        const float e1 = exp2_fast(d);
        kn[j] = kv[j] * exp2_fast(-d);
        qv[j] *= e1;
        kv[j] *= e1;
      }
      uint4 hi, lo;
      split8(qv, hi, lo);
      *reinterpret_cast<uint4*>(smem + pOffQKH + pan + o1) = hi;
      *reinterpret_cast<uint4*>(smem + pOffQKL + pan + o1) = lo;
      split8(kv, hi, lo);
      *reinterpret_cast<uint4*>(smem + pOffQKH + pan + o2) = hi;
      *reinterpret_cast<uint4*>(smem + pOffQKL + pan + o2) = lo;
      split8(kn, hi, lo);
      *reinterpret_cast<uint4*>(smem + pOffKNH + pan64 + o1) = hi;
      *reinterpret_cast<uint4*>(smem + pOffKNL + pan64 + o1) = lo;
    }
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = tmem_base_s;
  // 4. save the operand images; both score tiles in one M = 128 product: rows 0-63 Qp Kn^T, rows 64-127 Kp Kn^T
  if (tid == kLeaderK) {
    const Operand aH{sb + pOffQKH, 16384, 0}, aL{sb + pOffQKL, 16384, 0};
    const Operand bH{sb + pOffKNH, 8192, 0}, bL{sb + pOffKNL, 8192, 0};
    mma_tile(tbase, aH, bH, 128, 64, 8, false);
    mma_tile(tbase, aH, bL, 128, 64, 8, true);
    mma_tile(tbase, aL, bH, 128, 64, 8, true);
    mma_commit(&bar);
    bulk_store(p.kn_img + cidx * kKdaKnImg, sb + pOffKNH, 32768);
    bulk_commit();
  } else if (tid == 0) {
    bulk_store(p.qk_img + cidx * kKdaQkImg, sb + pOffQKH, 65536);
    bulk_commit();
  }
  // requested before the product is waited for
  const float bi = (quad >= 2 && tok < rows) ? ld_scalar(p.beta, (tok0 + tok) * p.beta_st + hv, p.beta_is_f32) : 0.f;
  const bool more = tile + gridDim.x < tiles;
  if (more) cur = tile_at(tile + gridDim.x);
  const bool ok = mbar_wait(&bar, parity, p.status, FLA_ERR_TIMEOUT);
  tc_fence_after();
  float sc[16];
  tmem_ld16(tmem_addr(tbase, quad * 32, j0), sc);
  tmem_ld_wait();
  tc_fence_before();
  if (quad < 2) {
    // 5a. q-side rows (eight warps): P = tril(Aqk) as split panels, then the next tile's loads
    if (tid == 0) bulk_wait_read();
    tri_sync<256>(2);
    uint8_t* img = smem + kStageP;
#pragma unroll
    for (int jj = 0; jj < 16; ++jj) sc[jj] = (ok && j0 + jj <= tok) ? sc[jj] : 0.f;   // select: masked entries may be inf
#pragma unroll
    for (int ch = 0; ch < 2; ++ch) {
      uint4 hi, lo;
      split8(sc + ch * 8, hi, lo);
      const uint32_t off = panel_chunk_off(tok, j0 / 8 + ch);
      *reinterpret_cast<uint4*>(img + off) = hi;
      *reinterpret_cast<uint4*>(img + 8192 + off) = lo;
    }
    fence_async_smem();
    tri_sync<256>(2);
    if (tid == 0) {
      bulk_store(p.p_img + cidx * kKdaPImg, sb + kStageP, 16384);
      bulk_commit();
      if (more) load_qk(cur);
    }
    if (more) {      // the gates of the next tile as far as L2: four threads a row, 128 bytes each
      const int t = (warp >> 2) * 64 + (warp & 1) * 32 + lane, es = p.g_is_f32 ? 4 : 2;
      if (t / 4 < cur.rows && (t & 3) * 128 < kK * es)
        prefetch_l2(static_cast<const char*>(p.g) + ((int64_t(cur.tok0) + t / 4) * p.g_st + cur.hv * p.g_sh) * es + (t & 3) * 128);
    }
  } else {
    // 5b. k-side rows (eight warps): Akk^T = (beta_i Kp Kn^T)^T, inverted where Kn was
    const int t = (warp >> 2) * 64 + (warp & 1) * 32 + lane;
    float* at = reinterpret_cast<float*>(smem + kStageA);
    if (tid == kLeaderK) bulk_wait_read();
    tri_sync<256>(1);
#pragma unroll
    for (int jj = 0; jj < 16; ++jj) {
      const int j = j0 + jj;
      at[j * kTriStride + tok] = ok && j < tok ? bi * sc[jj] : 0.f;      // select: entries above the diagonal may be inf
    }
    tri_sync<256>(1);
    tri_invert<256>(at, t, 1);
    tri_store_panels<256>(at, smem + kStageX, rows, t);
    fence_async_smem();
    tri_sync<256>(1);
    if (tid == kLeaderK) {
      bulk_store(p.x_img + cidx * kKdaXImg, sb + kStageX, 16384);
      bulk_commit();
    }
  }
  }
  if (tid == 0 || tid == kLeaderK) bulk_wait_read();     // the end of the kernel completes the writes
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base_s, 64);
}

// The two 64 x 64 score blocks of every chunk as plain tensors, for callers of the reference's low-level forward
// (npu_chunk_kda_fwd returns them): Aqk = scale tril(q k^T 2^{gk_i - gk_j}) from the P image and Akk = the chunk inverse
// from the X image (value + residual panels summed), rows and columns past a short chunk as zeros.
struct KdaExportParams {
  const bf16* img[2];
  void* out[2];
  int is_f32[2];
  int64_t sb[2], st[2], sh[2];
  const int32_t* cu_seqlens;
  const int32_t* chunk_offsets;
  int T, HV;
  float scale;
};
__global__ void __launch_bounds__(128) kda_export_scores_kernel(KdaExportParams p) {
  const int n = blockIdx.z, hv = blockIdx.y, c = blockIdx.x;
  const SeqInfo sq = seq_info(p.cu_seqlens, p.chunk_offsets, n, p.T);
  if (c >= sq.nt) return;
  const int rows = min(kC, sq.len - c * kC);
  const int64_t b = p.cu_seqlens ? 0 : n;
  const int64_t t0 = (p.cu_seqlens ? sq.bos : 0) + c * kC;
  const int64_t cidx = (int64_t(sq.cbase) + c) * p.HV + hv;
  for (int which = 0; which < 2; ++which) {
    if (!p.out[which]) continue;
    const uint8_t* hi = reinterpret_cast<const uint8_t*>(p.img[which] + cidx * 8192);
    const uint8_t* lo = hi + 8192;
    const float f = which ? 1.f : p.scale;
    for (int idx = threadIdx.x; idx < kC * 8; idx += 128) {
      const int r = idx >> 3, ch = idx & 7;
      if (r >= rows) continue;
      float a[8], l[8];
      unpack_bf16x8(*reinterpret_cast<const uint4*>(hi + panel_chunk_off(r, ch)), a);
      unpack_bf16x8(*reinterpret_cast<const uint4*>(lo + panel_chunk_off(r, ch)), l);
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] = (ch * 8 + j < rows && ch * 8 + j <= r) ? f * (a[j] + l[j]) : 0.f;
      const int64_t off = b * p.sb[which] + (t0 + r) * p.st[which] + hv * p.sh[which] + ch * 8;
      if (p.is_f32[which]) {
        float* dst = static_cast<float*>(p.out[which]) + off;
        *reinterpret_cast<float4*>(dst) = make_float4(a[0], a[1], a[2], a[3]);
        *reinterpret_cast<float4*>(dst + 4) = make_float4(a[4], a[5], a[6], a[7]);
      } else {
        *reinterpret_cast<uint4*>(static_cast<bf16*>(p.out[which]) + off) = pack8(a);
      }
    }
  }
}

}  // namespace fla

using namespace fla;

uint64_t fla::kda_ws_layout(int64_t total_chunks, int64_t HV, uint64_t off[5]) {
  uint64_t o = 256;
  const uint64_t per = uint64_t(total_chunks) * HV;
  off[0] = o; o += align_up(per * kKdaQkImg * 2, 256);
  off[1] = o; o += align_up(per * kKdaKnImg * 2, 256);
  off[2] = o; o += align_up(per * kKdaPImg * 2, 256);
  off[3] = o; o += align_up(per * kKdaXImg * 2, 256);
  off[4] = o; o += align_up(per * kKdaVecs * kK * 4, 256);
  return o;
}

uint64_t fla::kda_saved_layout(int64_t total_chunks, int64_t HV, int64_t nvb, int64_t tokens, int64_t segments, uint64_t off[5]) {
  uint64_t fo[5];
  const uint64_t per = uint64_t(total_chunks) * HV;
  uint64_t o = 0;
  off[0] = o; o += align_up(kda_ws_layout(total_chunks, HV, fo), 256);
  off[1] = o; o += align_up(uint64_t(tokens) * HV * kK * 4, 256);
  off[2] = o; o += align_up(per * nvb * kKdaSImg * 2, 256);
  off[3] = o; o += align_up(per * nvb * kKdaVnImg * 2, 256);
  off[4] = o; o += uint64_t(segments) * HV * kSegMBytes;
  return o;
}

static int kda_geometry(const fla_kda_chunk_fwd_args* a, int64_t* total_chunks, int* N, int* max_len) {
  const fla_tensor_t& q = a->q;
  if (!q.data || q.ndim != 4 || !a->v.data || a->v.ndim != 4) return FLA_ERR_SHAPE;
  const int64_t B = q.shape[0], T = q.shape[1];
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

static SegPlan kda_plan(const fla_kda_chunk_fwd_args* a, int64_t total_chunks, int N, int max_len) {
  return scan_plan(N, total_chunks, max_len, a->cu_seqlens.data != nullptr, a->v.shape[2], a->v.shape[3]);
}
// Operand images (unless they go into `saved`), then H and (again unless saved) M of the segments of split chains.
static uint64_t kda_fwd_workspace(const fla_kda_chunk_fwd_args* a, int64_t total_chunks, const SegPlan& plan) {
  uint64_t off[5];
  uint64_t b = a->saved.data ? 256 : kda_ws_layout(total_chunks, a->v.shape[2], off);
  if (plan.split) b += uint64_t(plan.count) * a->v.shape[2] * (kSegHBytes * (a->v.shape[3] / 128) + (a->saved.data ? 0 : kSegMBytes));
  return b;
}

extern "C" FLA_API int fla_b200_kda_chunk_fwd_workspace_size(const fla_kda_chunk_fwd_args* a, uint64_t* bytes) {
  if (!a || !bytes) return FLA_ERR_NULL;
  int64_t total_chunks; int N, max_len;
  const int st = kda_geometry(a, &total_chunks, &N, &max_len);
  if (st) return st;
  *bytes = kda_fwd_workspace(a, total_chunks, kda_plan(a, total_chunks, N, max_len));
  return FLA_OK;
}

extern "C" FLA_API int fla_b200_kda_chunk_saved_size(const fla_kda_chunk_fwd_args* a, uint64_t* bytes) {
  if (!a || !bytes) return FLA_ERR_NULL;
  int64_t total_chunks; int N, max_len;
  const int st = kda_geometry(a, &total_chunks, &N, &max_len);
  if (st) return st;
  uint64_t off[5];
  const int64_t V = a->v.shape[3];
  if (V != kV && V != 2 * kV) return FLA_ERR_SHAPE;
  const SegPlan plan = kda_plan(a, total_chunks, N, max_len);
  *bytes = kda_saved_layout(total_chunks, a->v.shape[2], V / kBV, a->q.shape[0] * a->q.shape[1], plan.split ? plan.count : 0, off);
  return FLA_OK;
}

static int kda_check_tok(const fla_tensor_t& t, int64_t B, int64_t T, int64_t heads, int64_t dim, bool allow_f32) {
  if (!t.data) return FLA_ERR_NULL;
  if (t.ndim != 4 || t.shape[0] != B || t.shape[1] != T || t.shape[2] != heads || t.shape[3] != dim) return FLA_ERR_SHAPE;
  if (t.dtype != FLA_BF16 && !(allow_f32 && t.dtype == FLA_F32)) return FLA_ERR_DTYPE;
  const int64_t esz = t.dtype == FLA_F32 ? 4 : 2;
  if (t.stride[3] != 1 || (t.stride[2] * esz) % 16 || (t.stride[1] * esz) % 16 || !aligned16(t.data)) return FLA_ERR_LAYOUT;
  if (B > 1 && t.stride[0] != T * t.stride[1]) return FLA_ERR_LAYOUT;
  return FLA_OK;
}

int fla::kda_check_rstd(const fla_tensor_t& q, const fla_tensor_t& k, int64_t B, int64_t T, int64_t HK) {
  if (!q.data && !k.data) return FLA_OK;
  for (const fla_tensor_t* t : {&q, &k}) {
    if (!t->data) return FLA_ERR_NULL;
    if (t->dtype != FLA_F32) return FLA_ERR_DTYPE;
    if (t->ndim != 3 || t->shape[0] != B || t->shape[1] != T || t->shape[2] != HK) return FLA_ERR_SHAPE;
    if (t->stride[2] != 1 || t->stride[1] != HK || (B > 1 && t->stride[0] != T * HK)) return FLA_ERR_LAYOUT;
  }
  return FLA_OK;
}

extern "C" FLA_API int fla_b200_kda_chunk_fwd(const fla_kda_chunk_fwd_args* a, void* workspace, uint64_t workspace_bytes,
                                              void* stream) {
  if (!a) return FLA_ERR_NULL;
  int64_t total_chunks; int N, max_len;
  int st = kda_geometry(a, &total_chunks, &N, &max_len);
  if (st) return st;
  const int64_t B = a->q.shape[0], T = a->q.shape[1], HK = a->q.shape[2], HV = a->v.shape[2];
  if (HK <= 0 || HV <= 0 || HV % HK) return FLA_ERR_SHAPE;
  const int64_t V = a->v.shape[3];
  if (V != kV && V != 2 * kV) return FLA_ERR_SHAPE;
  if ((st = kda_check_tok(a->q, B, T, HK, kK, false))) return st;
  if ((st = kda_check_tok(a->k, B, T, HK, kK, false))) return st;
  if ((st = kda_check_tok(a->v, B, T, HV, V, false))) return st;
  if ((st = kda_check_tok(a->g, B, T, HV, kK, true))) return st;
  if ((st = kda_check_tok(a->o, B, T, HV, V, true))) return st;
  const fla_tensor_t& be = a->beta;
  if (!be.data) return FLA_ERR_NULL;
  if (be.ndim != 3 || be.shape[0] != B || be.shape[1] != T || be.shape[2] != HV || be.stride[2] != 1 ||
      (B > 1 && be.stride[0] != T * be.stride[1]))
    return FLA_ERR_SHAPE;
  if (be.dtype != FLA_F32 && be.dtype != FLA_BF16) return FLA_ERR_DTYPE;
  for (const fla_tensor_t* s : {&a->initial_state, &a->final_state}) {
    if (!s->data) continue;
    if (s->dtype != FLA_F32) return FLA_ERR_DTYPE;
    if (s->ndim != 4 || s->shape[0] != N || s->shape[1] != HV || s->shape[2] != kK || s->shape[3] != V) return FLA_ERR_SHAPE;
    if (s->stride[3] != 1 || s->stride[2] != V || s->stride[1] != kK * V || s->stride[0] != HV * kK * V || !aligned16(s->data))
      return FLA_ERR_LAYOUT;
  }
  if (a->gate_mode < 0 || a->gate_mode > 2) return FLA_ERR_VALUE;
  if (a->gate_mode) {
    if (!a->a_log.data || a->a_log.dtype != FLA_F32 || a->a_log.ndim != 1 || a->a_log.shape[0] != HV || a->a_log.stride[0] != 1)
      return FLA_ERR_SHAPE;
    if (a->dt_bias.data && (a->dt_bias.dtype != FLA_F32 || a->dt_bias.ndim != 2 || a->dt_bias.shape[0] != HV ||
                            a->dt_bias.shape[1] != kK || a->dt_bias.stride[1] != 1 || a->dt_bias.stride[0] != kK))
      return FLA_ERR_SHAPE;
  }
  if (a->gk.data) {
    const fla_tensor_t& gk = a->gk;
    if (gk.dtype != FLA_F32 || gk.ndim != 4 || gk.shape[0] != B || gk.shape[1] != T || gk.shape[2] != HV || gk.shape[3] != kK ||
        gk.stride[3] != 1 || gk.stride[2] != kK || gk.stride[1] != HV * kK || (B > 1 && gk.stride[0] != T * HV * kK))
      return FLA_ERR_SHAPE;
  }
  if ((st = kda_check_rstd(a->q_rstd, a->k_rstd, B, T, HK))) return st;
  if (a->chunk_size != kC) return FLA_ERR_VALUE;
  uint64_t off[5];
  kda_ws_layout(total_chunks, HV, off);
  const SegPlan plan = kda_plan(a, total_chunks, N, max_len);
  const uint64_t need = kda_fwd_workspace(a, total_chunks, plan);
  uint8_t* images = static_cast<uint8_t*>(workspace);   // where the operand images go
  uint64_t soff[5] = {};
  if (a->saved.data) {
    const uint64_t sbytes = kda_saved_layout(total_chunks, HV, V / kBV, B * T, plan.split ? plan.count : 0, soff);
    if (a->saved.dtype != FLA_BF16 || a->saved.ndim != 1 || uint64_t(a->saved.shape[0]) * 2 < sbytes || !aligned16(a->saved.data))
      return FLA_ERR_SHAPE;
    if (a->gate_mode != 0 || a->gk.data) return FLA_ERR_VALUE;
    images = static_cast<uint8_t*>(a->saved.data) + soff[0];
  }
  if (!workspace || workspace_bytes < need || !aligned16(workspace)) return FLA_ERR_WORKSPACE;

  KdaParams p{};
  p.q = static_cast<const bf16*>(a->q.data); p.k = static_cast<const bf16*>(a->k.data); p.v = static_cast<const bf16*>(a->v.data);
  p.g = a->g.data; p.beta = be.data;
  p.a_log = static_cast<const float*>(a->a_log.data); p.dt_bias = static_cast<const float*>(a->dt_bias.data);
  p.q_rstd = static_cast<float*>(a->q_rstd.data); p.k_rstd = static_cast<float*>(a->k_rstd.data);
  p.gk_out = static_cast<float*>(a->gk.data);
  uint8_t* ws = images;
  p.status = reinterpret_cast<int*>(workspace);
  if (a->saved.data) {
    uint8_t* sv = static_cast<uint8_t*>(a->saved.data);
    p.gk_out = reinterpret_cast<float*>(sv + soff[1]);
    p.s_img = reinterpret_cast<bf16*>(sv + soff[2]);
    p.vn_img = reinterpret_cast<bf16*>(sv + soff[3]);
  }
  p.qk_img = reinterpret_cast<bf16*>(ws + off[0]); p.kn_img = reinterpret_cast<bf16*>(ws + off[1]);
  p.p_img = reinterpret_cast<bf16*>(ws + off[2]); p.x_img = reinterpret_cast<bf16*>(ws + off[3]);
  p.vec = reinterpret_cast<float*>(ws + off[4]);
  p.seg_len = plan.len;
  if (plan.split) {
    uint8_t* end = static_cast<uint8_t*>(workspace) + need - uint64_t(plan.count) * HV * kSegHBytes * (V / 128);
    p.seg_h = reinterpret_cast<float*>(end);
    p.seg_m = reinterpret_cast<bf16*>(a->saved.data ? static_cast<uint8_t*>(a->saved.data) + soff[4] : end - uint64_t(plan.count) * HV * kSegMBytes);
  }
  p.h0 = static_cast<const float*>(a->initial_state.data); p.ht = static_cast<float*>(a->final_state.data);
  p.o = a->o.data;
  p.cu_seqlens = static_cast<const int32_t*>(a->cu_seqlens.data);
  p.chunk_offsets = static_cast<const int32_t*>(a->chunk_offsets.data);
  p.q_st = a->q.stride[1]; p.q_sh = a->q.stride[2]; p.k_st = a->k.stride[1]; p.k_sh = a->k.stride[2];
  p.v_st = a->v.stride[1]; p.v_sh = a->v.stride[2]; p.o_st = a->o.stride[1]; p.o_sh = a->o.stride[2];
  p.g_st = a->g.stride[1]; p.g_sh = a->g.stride[2]; p.beta_st = be.stride[1];
  p.N = N; p.T = int(T); p.HK = int(HK); p.HV = int(HV); p.total_tokens = B * T; p.V = int(V); p.nvb = int(V / kBV);
  p.g_is_f32 = a->g.dtype == FLA_F32; p.beta_is_f32 = be.dtype == FLA_F32; p.o_is_f32 = a->o.dtype == FLA_F32;
  p.gate_mode = a->gate_mode; p.scale = a->scale; p.lower_bound = a->lower_bound;

  KdaExportParams ep{};
  for (int which = 0; which < 2; ++which) {
    const fla_tensor_t& t = which ? a->akk : a->aqk;
    if (!t.data) continue;
    if (t.ndim != 4 || t.shape[0] != B || t.shape[1] != T || t.shape[2] != HV || t.shape[3] != kC) return FLA_ERR_SHAPE;
    if (t.dtype != FLA_BF16 && t.dtype != FLA_F32) return FLA_ERR_DTYPE;
    if (t.stride[3] != 1 || !aligned16(t.data) || (t.stride[0] % 8) || (t.stride[1] % 8) || (t.stride[2] % 8)) return FLA_ERR_LAYOUT;
    ep.out[which] = t.data; ep.is_f32[which] = t.dtype == FLA_F32;
    ep.sb[which] = t.stride[0]; ep.st[which] = t.stride[1]; ep.sh[which] = t.stride[2];
  }

  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  const int nt_max = (max_len + kC - 1) / kC;
  st = kda_launch_forward(p, total_chunks, plan.count, cs);
  if (st || (!ep.out[0] && !ep.out[1])) return st;
  ep.img[0] = p.p_img; ep.img[1] = p.x_img;
  ep.cu_seqlens = p.cu_seqlens; ep.chunk_offsets = p.chunk_offsets; ep.T = p.T; ep.HV = p.HV; ep.scale = p.scale;
  KernelTimer kt("kda_export_scores", cs);
  kda_export_scores_kernel<<<dim3(nt_max, unsigned(p.HV), p.N), 128, 0, cs>>>(ep);
  return cuda_status(cudaGetLastError());
}

int fla::kda_launch_forward(const KdaParams& p, int64_t total_chunks, int64_t segments, cudaStream_t cs) {
  static std::atomic<bool> attr_done_dev[64] = {};   // per device ordinal; setting the attributes twice is harmless
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return FLA_ERR_CUDA;
  if (!attr_done_dev[dev]) {
    if (cudaFuncSetAttribute(kda_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kKdaPrepSmem) + 1024) != cudaSuccess) return FLA_ERR_CUDA;
    for (auto* scan : {kda_scan_fwd_kernel<false, false, false>, kda_scan_fwd_kernel<true, false, false>, kda_scan_fwd_kernel<false, false, true>,
                       kda_scan_fwd_kernel<true, false, true>, kda_scan_fwd_kernel<false, true, true>})
      if (cudaFuncSetAttribute(scan, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kKdaScanFwdSmem) + 1024) != cudaSuccess) return FLA_ERR_CUDA;
    attr_done_dev[dev] = true;
  }
  CUtensorMap tm_q, tm_k, tm_v;
  if (make_row_tile_map(&tm_v, p.v, uint64_t(p.V), uint64_t(p.HV), uint64_t(p.total_tokens), uint64_t(p.v_sh), uint64_t(p.v_st)) ||
      make_row_tile_map(&tm_q, p.q, kK, uint64_t(p.HK), uint64_t(p.total_tokens), uint64_t(p.q_sh), uint64_t(p.q_st)) ||
      make_row_tile_map(&tm_k, p.k, kK, uint64_t(p.HK), uint64_t(p.total_tokens), uint64_t(p.k_sh), uint64_t(p.k_st)))
    return FLA_ERR_CUDA;
  {
    KernelTimer kt("kda_prep", cs);
    const unsigned tiles = unsigned(total_chunks) * unsigned(p.HV);
    if (launch_pdl(kda_prep_kernel, std::min(tiles, 2u * unsigned(current_sm_count())), kKdaPrepThreads, kKdaPrepSmem + 1024, cs, p, tiles, tm_q, tm_k) != cudaSuccess)
      return FLA_ERR_CUDA;
  }
  {
    KernelTimer kt("kda_fwd", cs);
    const bool split = p.seg_len != kWholeSequence;
    const unsigned heads = unsigned(p.HV * (p.V / 128));
    if (split && launch_pdl(kda_scan_fwd_kernel<false, true, true>, dim3(heads, unsigned(segments), 2), kFwdThreads, kKdaScanFwdSmem + 1024, cs, p, tm_v) != cudaSuccess)
      return FLA_ERR_CUDA;
    auto* scan = split ? (p.s_img ? kda_scan_fwd_kernel<true, false, true> : kda_scan_fwd_kernel<false, false, true>)
                       : (p.s_img ? kda_scan_fwd_kernel<true, false, false> : kda_scan_fwd_kernel<false, false, false>);
    return cuda_status(launch_pdl(scan, dim3(heads, unsigned(segments)), kFwdThreads, kKdaScanFwdSmem + 1024, cs, p, tm_v));
  }
}
