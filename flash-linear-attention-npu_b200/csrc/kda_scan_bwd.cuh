// Reverse scan of the chunked KDA backward, the state gradient transposed in tensor memory (scan_common.cuh, kda_scan_fwd.cuh): one CTA per
// (sequence, value head, 128 channels of V).  Per chunk, last to first, with dS' the gradient entering from the right:
//     dS'a^T = dS'^T diag(e^{gk_L-a})              a factor per column, applied as the gradient is published
//     dVn^T  = scale dO^T P + dS'a^T Kn^T          zero past the end of the sequence
//     dZ^T   = dVn^T X;   dV = beta dZ;   bz = sum_v dZ V (partial sums per 32 channels)
//     dSa^T += [scale dO^T | -beta dZ^T] [Qp; Kp]  N = 128 key dims, three passes;   dS^T = dSa^T diag(e^a)
// Saved for the chunk-parallel kernel as strips whose rows are value channels (the layouts of the GDN reverse scan):
//     ds_img  dS'a [64-channel half][value | residual][16 strips of 8 key dims][64 rows x 16 bytes]
//     dz_img  [64-channel half][dO^T | dZ^T | residual of dZ^T][8 strips of 8 tokens][64 rows x 16 bytes]
#pragma once
#include "scan_common.cuh"
#include "scan_segments.cuh"

namespace fla {

// tensor-memory columns (512 allocated)
constexpr uint32_t kuDS = 0;       // dSa^T fp32 accumulator (128 key dims)
constexpr uint32_t kuAh = 128;     // dS'a^T as A operand; later [scale dO^T | -beta dZ^T] (128 rows of [Qp; Kp])
constexpr uint32_t kuAl = 192;
constexpr uint32_t kuW = 256;      // dS'a^T Kn^T accumulator, later dZ^T
constexpr uint32_t kuU = 320;      // dO^T P accumulator, later dO^T (fp32)
constexpr uint32_t kuDVh = 384;    // dVn^T as A operand
constexpr uint32_t kuDVl = 416;
constexpr uint32_t kuVT = 448;     // V^T (fp32)

// shared memory; only dO exists twice: every other operand has one reader per chunk and is loaded again once that has completed
constexpr uint32_t kbQK = 0;                 // 64 KB
constexpr uint32_t kbKn = 65536;             // 32 KB
constexpr uint32_t kbX = 98304;              // 16 KB
constexpr uint32_t kbP = 114688;             // 16 KB
constexpr uint32_t kbV = 131072;             // 16 KB
constexpr uint32_t kbD = 147456;             // 2 x 16 KB: dO rows
constexpr uint32_t kbO = 180224;             // 16 KB: dV rows on their way out
constexpr uint32_t kbI = 196608;             // 8 KB: identity panel
constexpr uint32_t kKdaScanBwdSmem = 204800;

struct KdaScanBwdBars {
  uint64_t *mma_bar, *qk_bar, *kn_bar, *x_bar, *p_bar, *v_bar, *d_bar;   // d: two (step parity)
};
__device__ __forceinline__ bool kda_bwd_mma1(uint32_t tbase, uint32_t sb, int s, KdaScanBwdBars bars, int* status, bool dead, uint32_t lead) {
  const uint32_t ph = s & 1;
  tc_fence_after();
  if (!dead && !mbar_wait(bars.kn_bar, ph, status, FLA_ERR_TIMEOUT)) dead = true;
  const Operand nh{sb + kbKn, 8192, 0}, nl{sb + kbKn + 16384, 8192, 0};        // rows (tokens) are N, reduction over key dims
  mma_tile_ts(tbase + kuW, tbase + kuAh, nh, 64, 8, false, lead);
  mma_tile_ts(tbase + kuW, tbase + kuAl, nh, 64, 8, true, lead);
  mma_tile_ts(tbase + kuW, tbase + kuAh, nl, 64, 8, true, lead);
  if (!dead && !mbar_wait(&bars.d_bar[s & 1], (s >> 1) & 1, status, FLA_ERR_TIMEOUT)) dead = true;
  if (!dead && !mbar_wait(bars.p_bar, ph, status, FLA_ERR_TIMEOUT)) dead = true;
  const Operand dt{sb + kbD + (s & 1) * 16384, 8192, 1};                       // dO^T: M = 128 channels, reduction over tokens
  const Operand p_h{sb + kbP, 8192, 1}, p_l{sb + kbP + 8192, 8192, 1};          // columns of P are N, rows the reduction
  mma_tile(tbase + kuU, dt, p_h, 128, 64, 4, false, lead);
  mma_tile(tbase + kuU, dt, p_l, 128, 64, 4, true, lead);
  mma_commit(bars.mma_bar, lead);
  return dead;
}
template <bool kState>
__device__ __forceinline__ bool kda_bwd_mma2(uint32_t tbase, uint32_t sb, int s, KdaScanBwdBars bars, int* status, bool dead, uint32_t lead) {
  const uint32_t ph = s & 1;
  tc_fence_after();
  if (!dead && !mbar_wait(bars.x_bar, ph, status, FLA_ERR_TIMEOUT)) dead = true;
  const Operand xh{sb + kbX, 8192, 1}, xl{sb + kbX + 8192, 8192, 1};
  mma_tile_ts(tbase + kuW, tbase + kuDVh, xh, 64, 4, false, lead);
  mma_tile_ts(tbase + kuW, tbase + kuDVl, xh, 64, 4, true, lead);
  mma_tile_ts(tbase + kuW, tbase + kuDVh, xl, 64, 4, true, lead);
  const Operand id{sb + kbI, 8192, 0};
  const Operand dt{sb + kbD + (s & 1) * 16384, 8192, 1}, vt{sb + kbV, 8192, 1};
  mma_tile(tbase + kuU, dt, id, 128, 64, 4, false, lead);                      // dO^T, exact
  if (!kState) {
    if (!dead && !mbar_wait(bars.v_bar, ph, status, FLA_ERR_TIMEOUT)) dead = true;
    mma_tile(tbase + kuVT, vt, id, 128, 64, 4, false, lead);                   // V^T, exact
  }
  mma_commit(bars.mma_bar, lead);
  return dead;
}
__device__ __forceinline__ bool kda_bwd_mma3(uint32_t tbase, uint32_t sb, int s, KdaScanBwdBars bars, int* status, bool dead, uint32_t lead) {
  tc_fence_after();
  if (!dead && !mbar_wait(bars.qk_bar, s & 1, status, FLA_ERR_TIMEOUT)) dead = true;
  const Operand h{sb + kbQK, 16384, 1}, l{sb + kbQK + 32768, 16384, 1};        // [Qp; Kp] rows are the reduction, N = 128 key dims
  mma_tile_ts(tbase + kuDS, tbase + kuAh, h, 128, 8, true, lead);
  mma_tile_ts(tbase + kuDS, tbase + kuAl, h, 128, 8, true, lead);
  mma_tile_ts(tbase + kuDS, tbase + kuAh, l, 128, 8, true, lead);
  mma_commit(bars.mma_bar, lead);
  return dead;
}
// D^T = dS^T M, 64 start dims each into the accumulators of W and U; the image of M sits where [Qp; Kp] will be
__device__ __forceinline__ bool kda_bwd_walk(uint32_t tbase, uint32_t sb, uint64_t* m_bar, uint32_t ph, uint64_t* mma_bar, int* status, bool dead, uint32_t lead) {
  tc_fence_after();
  if (!dead && !mbar_wait(m_bar, ph, status, FLA_ERR_TIMEOUT)) dead = true;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const Operand mh{sb + kbQK + half * 32768, 1024, 3}, ml{sb + kbQK + half * 32768 + 16384, 1024, 3};
    const uint32_t d = tbase + kuW + half * 64;
    mma_tile_ts(d, tbase + kuAh, mh, 64, 8, false, lead);
    mma_tile_ts(d, tbase + kuAl, mh, 64, 8, true, lead);
    mma_tile_ts(d, tbase + kuAh, ml, 64, 8, true, lead);
  }
  mma_commit(mma_bar, lead);
  return dead;
}

// kState: dH of a segment only.  kSplit: chains are split.
template <bool kState, bool kSplit>
__global__ void __launch_bounds__(kScanThreads, 1) kda_scan_bwd_kernel(KdaBwdParams p, const __grid_constant__ CUtensorMap tm_v,
                                                                        const __grid_constant__ CUtensorMap tm_d) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ KdaFactors fac[3];
  __shared__ uint32_t tmem_base_s;
  __shared__ __align__(8) uint64_t mma_bar, m_bar, qk_bar, kn_bar, x_bar, p_bar, v_bar, d_bar[2], f_bar[3];

  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  pdl_trigger();
  pdl_wait();
  const int seg = blockIdx.y + p.n0, hv = blockIdx.x / (p.V / 128), vb = blockIdx.x % (p.V / 128);
  if (tid == 0) clear_status(p.status, p.clear && seg + blockIdx.x == 0 && (kState || !kSplit));   // the backward's first kernel
  if (tid == 0 && blockIdx.y + blockIdx.x == 0) *p.counter = 0;      // of the par kernel that follows
  SegPos pos;
  if (!segment_pos<kSplit>(p.cu_seqlens, p.chunk_offsets, p.N, p.T, p.seg_len, seg, pos, p.n0, p.n1)) return;
  if (kState && pos.s == 0) return;
  const SeqInfo& sq = pos.sq;
  const int n = pos.n, nt = pos.nt;
  const uint32_t sb = smem_u32(smem);

  if (warp == 0) {
    tmem_alloc(&tmem_base_s, 512);
    tmem_relinquish();
  }
  if (tid == 0) {
    for (uint64_t* bar : {&mma_bar, &m_bar, &qk_bar, &kn_bar, &x_bar, &p_bar, &v_bar, &d_bar[0], &d_bar[1], &f_bar[0], &f_bar[1], &f_bar[2]}) mbar_init(bar, 1);
    mbar_init_fence();
  }
  write_identity_panel(smem + kbI, tid, kScanThreads);
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = tmem_base_s;
  bool dead = false;
  // step s = 0, 1, ... handles chunk nt - 1 - s
  auto chunk_head = [&](int s) { return (int64_t(sq.cbase) + nt - 1 - s) * p.HV + hv; };

  if (warp == 8) {
    // ============================================================ helper warp: loads
    auto bulk = [&](uint32_t dst, const bf16* src, uint32_t bytes, uint64_t* bar) {
      mbar_arrive_expect_tx(bar, bytes);
      bulk_load(dst, src, bytes, bar);
    };
    auto rows_tile = [&](uint32_t dst, const CUtensorMap* map, int s, uint64_t* bar) {
      const int row0 = sq.bos + (nt - 1 - s) * kC;
      mbar_arrive_expect_tx(bar, 16384);
      tma_load_tile(dst, map, vb * 128, hv, row0, bar);
      tma_load_tile(dst + 8192, map, vb * 128 + 64, hv, row0, bar);
    };
    auto load_qk = [&](int s) { bulk(sb + kbQK, p.qk_img + chunk_head(s) * kKdaQkImg, 65536, &qk_bar); };
    auto load_first = [&](int s) {      // operands of the first product
      bulk(sb + kbKn, p.kn_img + chunk_head(s) * kKdaKnImg, 32768, &kn_bar);
      bulk(sb + kbP, p.p_img + chunk_head(s) * kKdaPImg, 16384, &p_bar);
    };
    auto load_second = [&](int s) {     // of the second
      bulk(sb + kbX, p.x_img + chunk_head(s) * kKdaXImg, 16384, &x_bar);
      if (!kState) rows_tile(sb + kbV, &tm_v, s, &v_bar);
    };
    auto load_do = [&](int s) { rows_tile(sb + kbD + (s & 1) * 16384, &tm_d, s, &d_bar[s & 1]); };
    auto load_factors = [&](int s) {
      if (s < nt) {
        mbar_arrive_expect_tx(&f_bar[s % 3], uint32_t(sizeof(KdaFactors)));
        bulk_load(smem_u32(&fac[s % 3]), p.vec + chunk_head(s) * kKdaVecs * kK, uint32_t(sizeof(KdaFactors)), &f_bar[s % 3]);
      }
    };
    if (lane == 0) {
      tma_prefetch_descriptor(&tm_v);
      tma_prefetch_descriptor(&tm_d);
      if (nt > 0) {
        load_do(0);
        load_first(0);
        load_second(0);
      }
      load_factors(0);
      load_factors(1);
    }
    __syncwarp();
    if (kSplit && !kState) {
      for (int i = pos.ns - 2; i > pos.s; --i) {
        if (lane == 0) bulk(sb + kbQK, p.seg_m + (int64_t(seg - pos.s + i) * p.HV + hv) * 32768, 65536, &m_bar);
        __syncwarp();
        scan_sync();
        scan_sync();
      }
    }
    scan_sync();
    for (int s = 0; s < nt; ++s) {
      scan_sync();                                          // sync 1: step s - 1's update has read [Qp; Kp]
      if (lane == 0) {
        load_qk(s);
        if (s + 1 < nt) load_do(s + 1);
        load_factors(s + 2);
      }
      __syncwarp();
      scan_sync();                                          // sync 2: the first product has read Kn and P
      if (lane == 0 && s + 1 < nt) load_first(s + 1);
      __syncwarp();
      scan_sync();                                          // sync 3: the second has read X and v
      if (lane == 0 && s + 1 < nt) load_second(s + 1);
      __syncwarp();
    }
    scan_sync();
    return;
  }

  // ================================================================ epilogue warps
  const KdaScanBwdBars bars{&mma_bar, &qk_bar, &kn_bar, &x_bar, &p_bar, &v_bar, d_bar};
  const int warp_u = __shfl_sync(0xffffffffu, warp, 0);
  const uint32_t tbase_u = __shfl_sync(0xffffffffu, tbase, 0), sb_u = __shfl_sync(0xffffffffu, sb, 0);
  const int quad = warp & 3, half = warp >> 2;
  const int vrow = quad * 32 + lane;
  const uint32_t tlane = tmem_addr(tbase, quad * 32, 0);
  const int t_lo = half * 32, k_lo = half * 64;
  uint32_t mphase = 0;
  auto seg_dh = [&](int i) -> float* {      // dH of segment i of my sequence, at my channel's first key dim
    return p.seg_dh + ((int64_t(seg - pos.s + i) * p.HV + hv) * (p.V / 128) + vb) * (kK * 128) + k_lo * 128 + vrow;
  };
  {
    const float* src = nullptr;
    int64_t ld = p.V;
    if (!kSplit || pos.s + 1 == pos.ns) {
      if (p.dht) src = p.dht + ((int64_t(n) * p.HV + hv) * kK + k_lo) * p.V + vb * 128 + vrow;
    } else if (!kState) {
      src = seg_dh(pos.ns - 1);
      ld = 128;
    }
#pragma unroll
    for (int part = 0; part < 4; ++part) {
      float s16[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) s16[i] = src ? src[int64_t(part * 16 + i) * ld] : 0.f;
      tmem_st16(tlane + kuDS + k_lo + part * 16, s16);
    }
    tmem_st_wait();
  }
  if (kSplit && !kState) {
    for (int i = pos.ns - 2; i > pos.s; --i) {              // dS <- M_i^T dS + dH_i
#pragma unroll 1
      for (int part = 0; part < 4; ++part) {
        float s16[16];
        uint32_t hi[8], lo[8];
        tmem_ld16(tlane + kuDS + k_lo + part * 16, s16);
        tmem_ld_wait();
        split16(s16, hi, lo);
        tmem_st8u(tlane + kuAh + half * 32 + part * 8, hi);
        tmem_st8u(tlane + kuAl + half * 32 + part * 8, lo);
      }
      tmem_st_wait();
      tc_fence_before();
      scan_sync();
      tc_fence_after();
      if (warp_u == 0) dead = kda_bwd_walk(tbase_u, sb_u, &m_bar, (pos.ns - 2 - i) & 1, &mma_bar, p.status, dead, elect_one());
      const float* src = seg_dh(i);
      float h[64];
#pragma unroll
      for (int k = 0; k < 64; ++k) h[k] = src[k * 128];
      wait_or_mark(&mma_bar, mphase, dead, p.status);
      tc_fence_after();
#pragma unroll
      for (int part = 0; part < 4; ++part) {
        float s16[16];
        tmem_ld16(tlane + kuW + k_lo + part * 16, s16);
        tmem_ld_wait();
#pragma unroll
        for (int k = 0; k < 16; ++k) s16[k] += h[part * 16 + k];
        tmem_st16(tlane + kuDS + k_lo + part * 16, s16);
      }
      tmem_st_wait();
      tc_fence_before();
      scan_sync();
    }
  }
  // dO rows past the end of the sequence belong to whatever follows in memory: zeroed in shared memory
  if (nt > 0 && sq.len - (nt - 1) * kC < kC) {
    const int rows = sq.len - (nt - 1) * kC;
    if (!mbar_wait(&d_bar[0], 0, p.status, FLA_ERR_TIMEOUT)) dead = true;
    for (int idx = tid; idx < (kC - rows) * 16; idx += kScanEpiThreads) {
      const int r = rows + idx / 16, pc = idx % 16;
      *reinterpret_cast<uint4*>(smem + kbD + (pc >> 3) * 8192 + panel_chunk_off(r, pc & 7)) = make_uint4(0, 0, 0, 0);
    }
    fence_async_smem();
  }
  scan_sync();

  float ov[32];      // dV rows: formed in the third epilogue, stored while the update runs
  auto store_dv = [&](int c) {
    const int rows = min(kC, sq.len - c * kC);
    const int64_t off = (int64_t(sq.bos) + c * kC) * p.dv_st + hv * p.dv_sh + vb * 128;
    void* g = p.dv_f32 ? static_cast<void*>(static_cast<float*>(p.dv) + off) : static_cast<void*>(static_cast<bf16*>(p.dv) + off);
    store_rows_transposed(smem + kbO, ov, g, p.dv_st, p.dv_f32 != 0, rows, half, vrow, tid);
  };

  for (int s = 0; s < nt; ++s) {
    const int c = nt - 1 - s;
    const KdaFactors& f = fac[s % 3];
    if (!dead && !mbar_wait(&f_bar[s % 3], (s / 3) & 1, p.status, FLA_ERR_TIMEOUT)) dead = true;   // requested two steps ago
    const int rows = min(kC, sq.len - c * kC);
    const int64_t cidx = chunk_head(s) * (p.V / 128) + vb;

    // ---- A: dS'a (the accumulator still lacks the previous step's e^a): operand, saved image and accumulator
    {
      const float* ea = fac[(s + 2) % 3].ea;
      uint8_t* s_row = reinterpret_cast<uint8_t*>(p.ds_img + cidx * 32768) + (vrow >> 6) * 32768 + (vrow & 63) * 16;
#pragma unroll 1
      for (int g4 = 0; g4 < 4; ++g4) {
        float s16[16];
        tmem_ld16(tlane + kuDS + k_lo + g4 * 16, s16);
        tmem_ld_wait();
#pragma unroll
        for (int i4 = 0; i4 < 16; i4 += 4) {
          const float4 m = *reinterpret_cast<const float4*>(&f.el[k_lo + g4 * 16 + i4]);
          if (s > 0) {
            const float4 e = *reinterpret_cast<const float4*>(&ea[k_lo + g4 * 16 + i4]);
            s16[i4] *= e.x; s16[i4 + 1] *= e.y; s16[i4 + 2] *= e.z; s16[i4 + 3] *= e.w;
          }
          s16[i4] *= m.x; s16[i4 + 1] *= m.y; s16[i4 + 2] *= m.z; s16[i4 + 3] *= m.w;
        }
        uint32_t hi[8], lo[8];
        split16(s16, hi, lo);
        tmem_st8u(tlane + kuAh + half * 32 + g4 * 8, hi);
        tmem_st8u(tlane + kuAl + half * 32 + g4 * 8, lo);
        tmem_st16(tlane + kuDS + k_lo + g4 * 16, s16);
        if (!kState) {
          uint8_t* dst = s_row + (half * 8 + g4 * 2) * 1024;
          *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
          *reinterpret_cast<uint4*>(dst + 1024) = make_uint4(hi[4], hi[5], hi[6], hi[7]);
          *reinterpret_cast<uint4*>(dst + 16384) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
          *reinterpret_cast<uint4*>(dst + 16384 + 1024) = make_uint4(lo[4], lo[5], lo[6], lo[7]);
        }
        group_fence();
      }
      tmem_st_wait();
    }
    tc_fence_before();
    scan_sync();                                   // sync 1
    tc_fence_after();
    if (warp_u == 0) dead = kda_bwd_mma1(tbase_u, sb_u, s, bars, p.status, dead, elect_one());
    wait_or_mark(&mma_bar, mphase, dead, p.status);
    tc_fence_after();

    // ---- B: dVn^T = scale U + W (zero past the end of the sequence) for my 32 tokens
    {
#pragma unroll 1
      for (int g = 0; g < 2; ++g) {
        float w1[16], u1[16];
        tmem_ld16(tlane + kuW + t_lo + g * 16, w1);
        tmem_ld16(tlane + kuU + t_lo + g * 16, u1);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) u1[i] = (t_lo + g * 16 + i < rows) ? p.scale * u1[i] + w1[i] : 0.f;
        uint32_t hi[8], lo[8];
        split16(u1, hi, lo);
        tmem_st8u(tlane + kuDVh + half * 16 + g * 8, hi);
        tmem_st8u(tlane + kuDVl + half * 16 + g * 8, lo);
        group_fence();
      }
      tmem_st_wait();
    }
    tc_fence_before();
    scan_sync();                                   // sync 2
    tc_fence_after();
    if (warp_u == 0) dead = kda_bwd_mma2<kState>(tbase_u, sb_u, s, bars, p.status, dead, elect_one());
    wait_or_mark(&mma_bar, mphase, dead, p.status);
    tc_fence_after();

    // ---- C: dZ^T -> dV rows, partial sums of dZ V, the [dO^T | dZ^T] image, the operand [scale dO^T | -beta dZ^T]
    {
      uint8_t* img = reinterpret_cast<uint8_t*>(p.dz_img + cidx * (2 * kDzHalf)) + (vrow >> 6) * (2 * kDzHalf) + (vrow & 63) * 16;
      float pr[32];
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        float dz[16], t16[16];
        tmem_ld16(tlane + kuW + t_lo + g * 16, dz);
        if (!kState) tmem_ld16(tlane + kuVT + t_lo + g * 16, t16);
        tmem_ld_wait();
        uint32_t w8[8];
        if (!kState) {
#pragma unroll
          for (int i = 0; i < 16; ++i) pr[g * 16 + i] = dz[i] * t16[i];
          uint32_t zl[8];
          split16(dz, w8, zl);
          *reinterpret_cast<uint4*>(img + 8192 + (half * 4 + g * 2) * 1024) = make_uint4(w8[0], w8[1], w8[2], w8[3]);
          *reinterpret_cast<uint4*>(img + 8192 + (half * 4 + g * 2 + 1) * 1024) = make_uint4(w8[4], w8[5], w8[6], w8[7]);
          *reinterpret_cast<uint4*>(img + 16384 + (half * 4 + g * 2) * 1024) = make_uint4(zl[0], zl[1], zl[2], zl[3]);
          *reinterpret_cast<uint4*>(img + 16384 + (half * 4 + g * 2 + 1) * 1024) = make_uint4(zl[4], zl[5], zl[6], zl[7]);
        }
#pragma unroll
        for (int i4 = 0; i4 < 16; i4 += 4) {
          const float4 b4 = *reinterpret_cast<const float4*>(&f.b[t_lo + g * 16 + i4]);
          ov[g * 16 + i4] = b4.x * dz[i4];         dz[i4] = -ov[g * 16 + i4];
          ov[g * 16 + i4 + 1] = b4.y * dz[i4 + 1]; dz[i4 + 1] = -ov[g * 16 + i4 + 1];
          ov[g * 16 + i4 + 2] = b4.z * dz[i4 + 2]; dz[i4 + 2] = -ov[g * 16 + i4 + 2];
          ov[g * 16 + i4 + 3] = b4.w * dz[i4 + 3]; dz[i4 + 3] = -ov[g * 16 + i4 + 3];
        }
        uint32_t hi[8], lo[8];
        split16(dz, hi, lo);                              // -beta dZ^T: rows 64..127 of the [Qp; Kp] reduction
        tmem_st8u(tlane + kuAh + 32 + half * 16 + g * 8, hi);
        tmem_st8u(tlane + kuAl + 32 + half * 16 + g * 8, lo);
        tmem_ld16(tlane + kuU + t_lo + g * 16, t16);      // dO^T
        tmem_ld_wait();
        if (!kState) {
          pack16(t16, w8);                                // exact: these are the bf16 inputs
          *reinterpret_cast<uint4*>(img + (half * 4 + g * 2) * 1024) = make_uint4(w8[0], w8[1], w8[2], w8[3]);
          *reinterpret_cast<uint4*>(img + (half * 4 + g * 2 + 1) * 1024) = make_uint4(w8[4], w8[5], w8[6], w8[7]);
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) t16[i] *= p.scale;
        split16(t16, hi, lo);                             // scale dO^T: rows 0..63 of the reduction
        tmem_st8u(tlane + kuAh + half * 16 + g * 8, hi);
        tmem_st8u(tlane + kuAl + half * 16 + g * 8, lo);
        group_fence();
      }
      tmem_st_wait();
      if (!kState) {      // sum over my warp's 32 channels of dZ V for each of my 32 tokens; lane l ends up with token t_lo + l
        const float bzsum = warp_transpose_reduce32(pr, lane);
        if (t_lo + lane < rows)
          p.bz[(int64_t(vb * 4 + quad) * p.total_tokens + int64_t(sq.bos) + c * kC + t_lo + lane) * p.HV + hv] = bzsum;
      }
    }
    tc_fence_before();
    scan_sync();                                   // sync 3
    tc_fence_after();
    if (warp_u == 0) dead = kda_bwd_mma3(tbase_u, sb_u, s, bars, p.status, dead, elect_one());
    if (!kState) store_dv(c);
    wait_or_mark(&mma_bar, mphase, dead, p.status);
    tc_fence_after();
  }

  float* dst = kState ? seg_dh(pos.s)
                      : p.dh0 && (!kSplit || pos.s == 0) ? p.dh0 + ((int64_t(n) * p.HV + hv) * kK + k_lo) * p.V + vb * 128 + vrow : nullptr;
  const int64_t ld = kState ? 128 : p.V;
  if (!dead && dst) {
    const float* ea = fac[(nt + 2) % 3].ea;
#pragma unroll
    for (int part = 0; part < 4; ++part) {
      float s16[16];
      tmem_ld16(tlane + kuDS + k_lo + part * 16, s16);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 16; ++i) dst[int64_t(part * 16 + i) * ld] = nt > 0 ? s16[i] * ea[k_lo + part * 16 + i] : s16[i];
    }
  }
  tc_fence_before();
  scan_sync();
  if (warp == 0) tmem_dealloc(tbase, 512);
}

}  // namespace fla
