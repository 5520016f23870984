// Forward scan of chunked KDA, with the state transposed in tensor memory like the GDN scans (scan_common.cuh): one CTA per (sequence,
// value head, 128 channels of V), TMEM lane v = value channel v.  Per chunk, on the anchored operands of the prep kernel
// (kda_chunk_fwd.cu; Qp, Kp, Kn, P, X each a bf16 value + residual), with S the state at chunk start:
//     Sa^T   = S^T diag(e^a)                       a factor per column (key dim), applied as the state is published
//     [QS^T | KS^T] = Sa^T [Qp; Kp]^T              N = 128 tokens, three passes
//     Z^T    = beta (V^T - KS^T)                   v_new^T = Z^T X^T
//     Sa^T  += v_new^T Kn                          N = 128 key dims, three passes;   S'^T = Sa^T diag(e^{gk_L-a})
//     o^T    = scale (QS^T + v_new^T P^T)
// The kernel this replaces split V in 64-column blocks over two CTAs and staged the state and v_new through shared-memory panels.
// What the scan waits for: the chain of the three products and their epilogues; 144 KB of operand images per chunk.
// Images for the backward are strips whose rows are value channels, as in the GDN scan (s_img holds Sa).
#pragma once
#include "kda_common.cuh"
#include "scan_common.cuh"
#include "scan_segments.cuh"

namespace fla {

// tensor-memory columns (512 allocated)
constexpr uint32_t kfST = 0;       // Sa^T fp32 accumulator (128 key dims)
constexpr uint32_t kfSAh = 128;    // Sa^T as A operand: 128 key dims packed in 64 columns; its residual
constexpr uint32_t kfSAl = 192;
constexpr uint32_t kfKQ = 256;     // [QS^T (64 tokens) | KS^T (64 tokens)]
constexpr uint32_t kfVN = 320;     // v_new^T accumulator, later v_new^T P^T: reuses the KS^T columns
constexpr uint32_t kfZAh = 384;    // Z^T, then v_new^T, as A operand
constexpr uint32_t kfZAl = 416;
constexpr uint32_t kfVT = 448;     // V^T (fp32, 64 columns)

// shared memory.  [Qp; Kp] and Kn exist once, each loaded again as soon as its only reader of a chunk has completed; the rest twice.
constexpr uint32_t ksQK = 0;              // 64 KB: [Qp; Kp] rows, value then residual, two 64-column panels of 128 rows each
constexpr uint32_t ksKn = 65536;          // 32 KB: Kn, value then residual, two panels of 64 rows
constexpr uint32_t ksX = 98304;           // 2 x 16 KB: value + residual panels
constexpr uint32_t ksP = 131072;          // 2 x 16 KB
constexpr uint32_t ksV = 163840;          // 2 x 16 KB: v rows, two panels of 64 rows
constexpr uint32_t ksO = 196608;          // 16 KB: output rows on their way out
constexpr uint32_t ksI = 212992;          // 8 KB: identity panel
constexpr uint32_t kKdaScanFwdSmem = 221184;
// the image of M during the walk: four pieces of 16 KB in Kn and the X, P buffers of odd chunks
__host__ __device__ constexpr uint32_t kda_walk_piece(int i) { return i < 2 ? ksKn + i * 16384 : i == 2 ? ksX + 16384 : ksP + 16384; }

struct KdaScanBars {
  uint64_t *mma_bar, *o_bar, *qk_bar, *kn_bar, *x_bar, *p_bar, *v_bar;   // x, p, v: two each (chunk parity)
};
template <bool kState>
__device__ __forceinline__ bool kda_fwd_mma1(uint32_t tbase, uint32_t sb, int c, KdaScanBars bars, bool values, int* status, bool dead, uint32_t lead) {
  const int b = c & 1;
  tc_fence_after();
  if (!dead && !mbar_wait(bars.qk_bar, c & 1, status, FLA_ERR_TIMEOUT)) dead = true;
  const uint32_t off = kState ? 8192 : 0, col = kState ? kfKQ + 64 : kfKQ;      // the state-only pass needs the Kp rows only
  const int n = kState ? 64 : 128;
  const Operand h{sb + ksQK + off, 16384, 0}, l{sb + ksQK + 32768 + off, 16384, 0};
  mma_tile_ts(tbase + col, tbase + kfSAh, h, n, 8, false, lead);
  mma_tile_ts(tbase + col, tbase + kfSAl, h, n, 8, true, lead);
  mma_tile_ts(tbase + col, tbase + kfSAh, l, n, 8, true, lead);
  if (!kState || values) {
    if (!dead && !mbar_wait(&bars.v_bar[b], (c >> 1) & 1, status, FLA_ERR_TIMEOUT)) dead = true;
    const Operand vt{sb + ksV + b * 16384, 8192, 1}, id{sb + ksI, 8192, 0};
    mma_tile(tbase + kfVT, vt, id, 128, 64, 4, false, lead);                     // V^T, exact
  }
  mma_commit(bars.mma_bar, lead);
  return dead;
}
__device__ __forceinline__ bool kda_fwd_mma2(uint32_t tbase, uint32_t sb, int c, KdaScanBars bars, int* status, bool dead, uint32_t lead) {
  const int b = c & 1;
  tc_fence_after();
  if (!dead && !mbar_wait(&bars.x_bar[b], (c >> 1) & 1, status, FLA_ERR_TIMEOUT)) dead = true;
  const Operand xh{sb + ksX + b * 16384, 8192, 0}, xl{sb + ksX + b * 16384 + 8192, 8192, 0};   // rows of X are N, columns the reduction
  mma_tile_ts(tbase + kfVN, tbase + kfZAh, xh, 64, 4, false, lead);
  mma_tile_ts(tbase + kfVN, tbase + kfZAl, xh, 64, 4, true, lead);
  mma_tile_ts(tbase + kfVN, tbase + kfZAh, xl, 64, 4, true, lead);
  mma_commit(bars.mma_bar, lead);
  return dead;
}
template <bool kState>
__device__ __forceinline__ bool kda_fwd_mma3(uint32_t tbase, uint32_t sb, int c, KdaScanBars bars, int* status, bool dead, uint32_t lead) {
  const int b = c & 1;
  tc_fence_after();
  if (!dead && !mbar_wait(bars.kn_bar, c & 1, status, FLA_ERR_TIMEOUT)) dead = true;
  const Operand nh{sb + ksKn, 8192, 1}, nl{sb + ksKn + 16384, 8192, 1};          // rows (tokens) are the reduction, N = 128 key dims
  mma_tile_ts(tbase + kfST, tbase + kfZAh, nh, 128, 4, true, lead);
  mma_tile_ts(tbase + kfST, tbase + kfZAl, nh, 128, 4, true, lead);
  mma_tile_ts(tbase + kfST, tbase + kfZAh, nl, 128, 4, true, lead);
  mma_commit(bars.mma_bar, lead);                                                // the state update: what the next chunk waits for
  if (kState) return dead;
  if (!dead && !mbar_wait(&bars.p_bar[b], (c >> 1) & 1, status, FLA_ERR_TIMEOUT)) dead = true;
  const Operand ph{sb + ksP + b * 16384, 8192, 0}, pl{sb + ksP + b * 16384 + 8192, 8192, 0};
  mma_tile_ts(tbase + kfVN, tbase + kfZAh, ph, 64, 4, false, lead);
  mma_tile_ts(tbase + kfVN, tbase + kfZAl, ph, 64, 4, true, lead);
  mma_tile_ts(tbase + kfVN, tbase + kfZAh, pl, 64, 4, true, lead);
  mma_commit(bars.o_bar, lead);
  return dead;
}
// D^T = S^T M^T (scan_segments.cuh)
__device__ __forceinline__ bool kda_fwd_walk(uint32_t tbase, uint32_t sb, uint64_t* m_bar, uint32_t ph, uint64_t* mma_bar, int* status, bool dead, uint32_t lead) {
  tc_fence_after();
  if (!dead && !mbar_wait(m_bar, ph, status, FLA_ERR_TIMEOUT)) dead = true;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const Operand mh{sb + kda_walk_piece(half * 2), 1024, 2}, ml{sb + kda_walk_piece(half * 2 + 1), 1024, 2};
    mma_tile_ts(tbase + kfKQ, tbase + kfSAh + half * 32, mh, 128, 4, half > 0, lead);
    mma_tile_ts(tbase + kfKQ, tbase + kfSAl + half * 32, mh, 128, 4, true, lead);
    mma_tile_ts(tbase + kfKQ, tbase + kfSAh + half * 32, ml, 128, 4, true, lead);
  }
  mma_commit(mma_bar, lead);
  return dead;
}
// kSave: also the images the backward reads.  kState: a segment's M (blockIdx.z = 1) or H (0) only.  kSplit: chains are split.
template <bool kSave, bool kState, bool kSplit>
__global__ void __launch_bounds__(kFwdThreads, 1) kda_scan_fwd_kernel(KdaParams p, const __grid_constant__ CUtensorMap tm_v) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ KdaFactors fac[3];
  __shared__ uint32_t tmem_base_s;
  __shared__ __align__(8) uint64_t mma_bar, o_bar, m_bar, qk_bar, kn_bar, x_bar[2], p_bar[2], v_bar[2], f_bar[3];

  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  pdl_trigger();
  pdl_wait();
  const int seg = blockIdx.y, hv = blockIdx.x / (p.V / 128), vb = blockIdx.x % (p.V / 128);
  SegPos pos;
  if (!segment_pos<kSplit>(p.cu_seqlens, p.chunk_offsets, p.N, p.T, p.seg_len, seg, pos, 0, p.N)) return;
  const bool values = blockIdx.z == 0;
  if (kState) {                                            // H of every segment but the last, M of those between the first and the last
    if (pos.s + 1 == pos.ns || (!values && (pos.s == 0 || vb > 0))) return;
  }
  const SeqInfo& sq = pos.sq;
  const int nt = pos.nt, n = pos.n;
  const uint32_t sb = smem_u32(smem);

  if (warp == 0) {
    tmem_alloc(&tmem_base_s, 512);
    tmem_relinquish();
  }
  if (tid == 0) {
    mbar_init(&mma_bar, 1);
    mbar_init(&o_bar, 1);
    mbar_init(&m_bar, 1);
    mbar_init(&qk_bar, 1);
    mbar_init(&kn_bar, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&x_bar[i], 1);
      mbar_init(&p_bar[i], 1);
      mbar_init(&v_bar[i], 1);
    }
    for (int i = 0; i < 3; ++i) mbar_init(&f_bar[i], 1);
    mbar_init_fence();
  }
  write_identity_panel(smem + ksI, tid, kFwdThreads);
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = tmem_base_s;
  bool dead = false;
  auto chunk_head = [&](int c) { return (int64_t(sq.cbase) + c) * p.HV + hv; };

  if (warp == kFwdEpiWarps) {
    // ============================================================ helper warp: loads
    auto load_qk = [&](int c) {
      mbar_arrive_expect_tx(&qk_bar, 65536);
      bulk_load(sb + ksQK, p.qk_img + chunk_head(c) * kKdaQkImg, 65536, &qk_bar);
    };
    auto load_kn = [&](int c) {
      mbar_arrive_expect_tx(&kn_bar, 32768);
      bulk_load(sb + ksKn, p.kn_img + chunk_head(c) * kKdaKnImg, 32768, &kn_bar);
    };
    auto load_rest = [&](int c) {
      const int b = c & 1, row0 = sq.bos + c * kC;
      if (!kState || values) {
        mbar_arrive_expect_tx(&v_bar[b], 16384);
        tma_load_tile(sb + ksV + b * 16384, &tm_v, vb * 128, hv, row0, &v_bar[b]);
        tma_load_tile(sb + ksV + b * 16384 + 8192, &tm_v, vb * 128 + 64, hv, row0, &v_bar[b]);
      }
      mbar_arrive_expect_tx(&x_bar[b], 16384);
      bulk_load(sb + ksX + b * 16384, p.x_img + chunk_head(c) * kKdaXImg, 16384, &x_bar[b]);
      if (!kState) {
        mbar_arrive_expect_tx(&p_bar[b], 16384);
        bulk_load(sb + ksP + b * 16384, p.p_img + chunk_head(c) * kKdaPImg, 16384, &p_bar[b]);
      }
    };
    auto load_factors = [&](int c) {
      if (c < nt) {
        mbar_arrive_expect_tx(&f_bar[c % 3], uint32_t(sizeof(KdaFactors)));
        bulk_load(smem_u32(&fac[c % 3]), p.vec + chunk_head(c) * kKdaVecs * kK, uint32_t(sizeof(KdaFactors)), &f_bar[c % 3]);
      }
    };
    if (lane == 0) {
      tma_prefetch_descriptor(&tm_v);
      if (nt > 0) {
        load_qk(0);
        load_rest(0);
      }
      load_factors(0);
      load_factors(1);
    }
    __syncwarp();
    if (kSplit && !kState) {      // the images of the earlier segments' M, one at a time
      for (int i = 1; i < pos.s; ++i) {
        if (lane == 0) {
          const bf16* img = p.seg_m + (int64_t(seg - pos.s + i) * p.HV + hv) * 32768;
          mbar_arrive_expect_tx(&m_bar, 65536);
#pragma unroll
          for (int piece = 0; piece < 4; ++piece) bulk_load(sb + kda_walk_piece(piece), img + piece * 8192, 16384, &m_bar);
        }
        __syncwarp();
        scan_sync();
        scan_sync();
      }
    }
    scan_sync();
    for (int c = 0; c < nt; ++c) {
      scan_sync();                                          // sync 1: chunk c - 1's state update has read Kn
      if (lane == 0) {
        load_kn(c);
        if (c + 1 < nt) load_rest(c + 1);
        load_factors(c + 2);
      }
      __syncwarp();
      scan_sync();                                          // sync 2: the first product of chunk c has read [Qp; Kp]
      if (lane == 0 && c + 1 < nt) load_qk(c + 1);
      __syncwarp();
      scan_sync();                                          // sync 3
    }
    scan_sync();
    return;
  }

  // ================================================================ epilogue warps
  const KdaScanBars bars{&mma_bar, &o_bar, &qk_bar, &kn_bar, x_bar, p_bar, v_bar};
  const int warp_u = __shfl_sync(0xffffffffu, warp, 0);
  const uint32_t tbase_u = __shfl_sync(0xffffffffu, tbase, 0), sb_u = __shfl_sync(0xffffffffu, sb, 0);
  const int quad = warp & 3, cs = warp >> 2;
  const int vrow = quad * 32 + lane;
  const uint32_t tlane = tmem_addr(tbase, quad * 32, 0);
  const int t_lo = cs * kFwdTT, k_lo = cs * kFwdKT;
  uint32_t mphase = 0, ophase = 0;

  {   // the state at the start of my segment (or the first segment's end, where the walk starts) into the accumulator columns
    const float* src = nullptr;
    int64_t ld = p.V;
    if (!kSplit || pos.s == 0) {
      if (p.h0) src = p.h0 + ((int64_t(n) * p.HV + hv) * kK + k_lo) * p.V + vb * 128 + vrow;
    } else if (!kState) {
      src = p.seg_h + ((int64_t(seg - pos.s) * p.HV + hv) * (p.V / 128) + vb) * (kK * 128) + k_lo * 128 + vrow;
      ld = 128;
    }
#pragma unroll
    for (int part = 0; part < kFwdKT / 16; ++part) {
      float s16[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) s16[i] = src ? src[int64_t(part * 16 + i) * ld] : 0.f;
      if (kState && !values) {
#pragma unroll
        for (int i = 0; i < 16; ++i) s16[i] = k_lo + part * 16 + i == vrow ? 1.f : 0.f;
      }
      tmem_st16(tlane + kfST + k_lo + part * 16, s16);
    }
    tmem_st_wait();
  }
  if (kSplit && !kState) {
    for (int i = 1; i < pos.s; ++i) {                       // S <- M_i S + H_i
#pragma unroll
      for (int part = 0; part < kFwdKT / 16; ++part) {
        float s16[16];
        uint32_t hi[8], lo[8];
        tmem_ld16(tlane + kfST + k_lo + part * 16, s16);
        tmem_ld_wait();
        split16(s16, hi, lo);
        tmem_st8u(tlane + kfSAh + cs * (kFwdKT / 2) + part * 8, hi);
        tmem_st8u(tlane + kfSAl + cs * (kFwdKT / 2) + part * 8, lo);
      }
      tmem_st_wait();
      tc_fence_before();
      scan_sync();
      tc_fence_after();
      if (warp_u == 0) dead = kda_fwd_walk(tbase_u, sb_u, &m_bar, (i - 1) & 1, &mma_bar, p.status, dead, elect_one());
      const float* src = p.seg_h + ((int64_t(seg - pos.s + i) * p.HV + hv) * (p.V / 128) + vb) * (kK * 128) + k_lo * 128 + vrow;
      float h[kFwdKT];
#pragma unroll
      for (int k = 0; k < kFwdKT; ++k) h[k] = src[k * 128];
      wait_or_mark(&mma_bar, mphase, dead, p.status);
      tc_fence_after();
#pragma unroll
      for (int part = 0; part < kFwdKT / 16; ++part) {
        float s16[16];
        tmem_ld16(tlane + kfKQ + k_lo + part * 16, s16);
        tmem_ld_wait();
#pragma unroll
        for (int k = 0; k < 16; ++k) s16[k] += h[part * 16 + k];
        tmem_st16(tlane + kfST + k_lo + part * 16, s16);
      }
      tmem_st_wait();
      tc_fence_before();
      scan_sync();
    }
  }
  scan_sync();

  float ov[kFwdTT];
  auto form_o = [&]() {
    float pv[16];
    tmem_ld16(tlane + kfKQ + t_lo, ov);
    tmem_ld16(tlane + kfVN + t_lo, pv);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 16; ++i) ov[i] = p.scale * (ov[i] + pv[i]);
  };
  static_assert(kFwdTT == 16, "a thread's tokens of a tile are one group");
  auto store_o = [&](int c) {
    if (!p.o) return;
    const int rows = min(kC, sq.len - c * kC);
    const int64_t off = (int64_t(sq.bos) + c * kC) * p.o_st + hv * p.o_sh + vb * 128;
    void* g = p.o_is_f32 ? static_cast<void*>(static_cast<float*>(p.o) + off) : static_cast<void*>(static_cast<bf16*>(p.o) + off);
    fwd_store_rows_transposed(smem + ksO, ov, g, p.o_st, p.o_is_f32 != 0, rows, cs, vrow, tid);
  };

  for (int c = 0; c < nt; ++c) {
    const KdaFactors& f = fac[c % 3];
    if (!dead && !mbar_wait(&f_bar[c % 3], (c / 3) & 1, p.status, FLA_ERR_TIMEOUT)) dead = true;   // requested two chunks ago
    const int rows = min(kC, sq.len - c * kC);
    const int64_t cidx = chunk_head(c) * (p.V / 128) + vb;

    // ---- A: Sa = diag(e^a) S (S still carries the previous chunk's e^{gk_L - a}): operand, saved image and accumulator
    {
      const float* el = fac[(c + 2) % 3].el;               // the previous chunk's record
      uint8_t* s_row = kSave ? reinterpret_cast<uint8_t*>(p.s_img + cidx * 32768) + (vrow >> 6) * 32768 + (vrow & 63) * 16 : nullptr;
#pragma unroll 1
      for (int g4 = 0; g4 < kFwdKT / 16; ++g4) {
        float s16[16];
        tmem_ld16(tlane + kfST + k_lo + g4 * 16, s16);
        tmem_ld_wait();
#pragma unroll
        for (int i4 = 0; i4 < 16; i4 += 4) {
          float4 m = *reinterpret_cast<const float4*>(&f.ea[k_lo + g4 * 16 + i4]);
          if (c > 0) {
            const float4 e = *reinterpret_cast<const float4*>(&el[k_lo + g4 * 16 + i4]);
            s16[i4] *= e.x; s16[i4 + 1] *= e.y; s16[i4 + 2] *= e.z; s16[i4 + 3] *= e.w;
          }
          s16[i4] *= m.x; s16[i4 + 1] *= m.y; s16[i4 + 2] *= m.z; s16[i4 + 3] *= m.w;
        }
        uint32_t hi[8], lo[8];
        split16(s16, hi, lo);
        tmem_st8u(tlane + kfSAh + cs * (kFwdKT / 2) + g4 * 8, hi);
        tmem_st8u(tlane + kfSAl + cs * (kFwdKT / 2) + g4 * 8, lo);
        tmem_st16(tlane + kfST + k_lo + g4 * 16, s16);
        if (kSave) {
          uint8_t* dst = s_row + (cs * (kFwdKT / 8) + g4 * 2) * 1024;
          *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
          *reinterpret_cast<uint4*>(dst + 1024) = make_uint4(hi[4], hi[5], hi[6], hi[7]);
          *reinterpret_cast<uint4*>(dst + 16384) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
          *reinterpret_cast<uint4*>(dst + 16384 + 1024) = make_uint4(lo[4], lo[5], lo[6], lo[7]);
        }
        group_fence();
      }
      tmem_st_wait();
    }
    if (!kState && c > 0) {   // the output accumulators of chunk c - 1: into registers before the next product overwrites them
      wait_or_mark(&o_bar, ophase, dead, p.status);
      tc_fence_after();
      form_o();
    }
    tc_fence_before();
    scan_sync();                                   // sync 1
    tc_fence_after();
    if (warp_u == 0) dead = kda_fwd_mma1<kState>(tbase_u, sb_u, c, bars, values, p.status, dead, elect_one());
    if (!kState && c > 0) store_o(c - 1);          // while [QS^T | KS^T] runs
    wait_or_mark(&mma_bar, mphase, dead, p.status);
    tc_fence_after();

    // ---- C: Z^T = beta (V^T - KS^T) for my 16 tokens
    {
      float ks[16], vt[16];
      tmem_ld16(tlane + kfKQ + 64 + t_lo, ks);
      if (!kState || values) {
        tmem_ld16(tlane + kfVT + t_lo, vt);
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) vt[i] = 0.f;
      }
      tmem_ld_wait();
#pragma unroll
      for (int i4 = 0; i4 < 16; i4 += 4) {
        const float4 b4 = *reinterpret_cast<const float4*>(&f.b[t_lo + i4]);
        ks[i4] = b4.x * (vt[i4] - ks[i4]);
        ks[i4 + 1] = b4.y * (vt[i4 + 1] - ks[i4 + 1]);
        ks[i4 + 2] = b4.z * (vt[i4 + 2] - ks[i4 + 2]);
        ks[i4 + 3] = b4.w * (vt[i4 + 3] - ks[i4 + 3]);
      }
      uint32_t hi[8], lo[8];
      split16(ks, hi, lo);
      tmem_st8u(tlane + kfZAh + cs * 8, hi);
      tmem_st8u(tlane + kfZAl + cs * 8, lo);
      tmem_st_wait();
    }
    tc_fence_before();
    scan_sync();                                   // sync 2
    tc_fence_after();
    if (warp_u == 0) dead = kda_fwd_mma2(tbase_u, sb_u, c, bars, p.status, dead, elect_one());
    wait_or_mark(&mma_bar, mphase, dead, p.status);
    tc_fence_after();

    // ---- E: v_new^T (rows past the end of the sequence are zero)
    {
      float vn[16];
      tmem_ld16(tlane + kfVN + t_lo, vn);
      tmem_ld_wait();
      if (rows < kC) {
#pragma unroll
        for (int i = 0; i < 16; ++i) vn[i] = t_lo + i < rows ? vn[i] : 0.f;
      }
      uint32_t hi[8], lo[8];
      split16(vn, hi, lo);
      tmem_st8u(tlane + kfZAh + cs * 8, hi);
      tmem_st8u(tlane + kfZAl + cs * 8, lo);
      if (kSave) {
        uint8_t* dst = reinterpret_cast<uint8_t*>(p.vn_img + cidx * 16384) + (vrow >> 6) * 16384 + cs * 2 * 1024 + (vrow & 63) * 16;
        *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(dst + 1024) = make_uint4(hi[4], hi[5], hi[6], hi[7]);
        *reinterpret_cast<uint4*>(dst + 8192) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        *reinterpret_cast<uint4*>(dst + 8192 + 1024) = make_uint4(lo[4], lo[5], lo[6], lo[7]);
      }
      tmem_st_wait();
    }
    tc_fence_before();
    scan_sync();                                   // sync 3
    tc_fence_after();
    if (warp_u == 0) dead = kda_fwd_mma3<kState>(tbase_u, sb_u, c, bars, p.status, dead, elect_one());
    wait_or_mark(&mma_bar, mphase, dead, p.status);    // the state update has completed (the output product may still run)
    tc_fence_after();
  }

  if (!kState && nt > 0) {
    wait_or_mark(&o_bar, ophase, dead, p.status);
    tc_fence_after();
    form_o();
    store_o(nt - 1);
  }
  float* dst = p.ht && (!kSplit || pos.s + 1 == pos.ns) ? p.ht + ((int64_t(n) * p.HV + hv) * kK + k_lo) * p.V + vb * 128 + vrow : nullptr;
  int64_t ld = p.V;
  if (kState) {
    dst = values ? p.seg_h + ((int64_t(seg) * p.HV + hv) * (p.V / 128) + vb) * (kK * 128) + k_lo * 128 + vrow : nullptr;
    ld = 128;
  }
  if (!dead && (dst || (kState && !values))) {
    const float* el = fac[(nt + 2) % 3].el;
#pragma unroll
    for (int part = 0; part < kFwdKT / 16; ++part) {
      float s16[16];
      tmem_ld16(tlane + kfST + k_lo + part * 16, s16);
      tmem_ld_wait();
      if (nt > 0) {
#pragma unroll
        for (int i = 0; i < 16; ++i) s16[i] *= el[k_lo + part * 16 + i];
      }
      if (kState && !values) {                     // M as an operand image, [64 start dims][value | residual][16 strips of 8 end dims]
        uint32_t hi[8], lo[8];
        split16(s16, hi, lo);
        uint8_t* img = reinterpret_cast<uint8_t*>(p.seg_m + (int64_t(seg) * p.HV + hv) * 32768) + (vrow >> 6) * 32768 + (vrow & 63) * 16 +
                       (k_lo / 8 + part * 2) * 1024;
        *reinterpret_cast<uint4*>(img) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(img + 1024) = make_uint4(hi[4], hi[5], hi[6], hi[7]);
        *reinterpret_cast<uint4*>(img + 16384) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        *reinterpret_cast<uint4*>(img + 16384 + 1024) = make_uint4(lo[4], lo[5], lo[6], lo[7]);
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) dst[int64_t(part * 16 + i) * ld] = s16[i];
      }
    }
  }
  tc_fence_before();
  scan_sync();
  if (warp == 0) tmem_dealloc(tbase, 512);
}

}  // namespace fla
