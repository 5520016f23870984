// Chunked gated-delta-rule backward (chunk = 64, K = V = 128) as two kernels.
//
// With per chunk  gam = cumsum(g),  P = tril(Q K^T * e^{gam_i-gam_j}),  X = (I + strict_tril(beta_i e^{gam_i-gam_j} k_i.k_j))^-1,
// S = state at chunk start, Vn = v_new (both saved by the forward as bf16 value + residual strip images) and dS' the state
// gradient entering the chunk from the right:
//
//  gdn_scan_bwd_kernel  (gdn_scan_bwd.cuh; reverse-sequential over chunks, one CTA per (sequence, value head, 128 channels of V)):
//      dVn = scale P^T dO + e^{gam_L-gam} * (K dS')          dZ = X^T dVn          dV = beta * dZ
//      dS  = e^{gam_L} dS' + (scale e^{gam} * Q)^T dO - K^T (beta e^{gam} * dZ)     dh0 = dS after the first chunk
//      saves dS' and [dO; dZ] as strip images and the partial row sums  sum_v dZ*V  for the second kernel.
//      Replaces chunk_bwd_dv_local + chunk_gated_delta_rule_bwd_dhu of the reference
//      (examples/flash_gated_delta_rule.py:930-960) and the dv / du parts of prepare_wy_repr_bwd_*.
//  gdn_bwd_par_kernel  (parallel over chunks, one CTA per (chunk, q/k head), looping over the value heads of the group):
//      dP  = scale tril(dO Vn^T * e^{gam_i-gam_j})            dA = -strict_tril(dZ Vn^T)       dAt = dA * beta_i e^{gam_i-gam_j}
//      dq  = scale e^{gam} * (dO S^T) + dP K
//      dk  = dP^T Q + dAt^T K + dAt K + e^{gam_L-gam} * (Vn dS'^T) - beta e^{gam} * (dZ S^T)
//      dbeta = sum_v dZ*V - e^{gam} k.(dZ S^T) + sum_j dA_ij e^{gam_i-gam_j} k_i.k_j
//      dgam  = q.dq - k.dk + 2 beta (sum_j dA_ij e^{..} k_i.k_j) - 2 beta e^{gam} k.(dZ S^T);
//      dgam_L += e^{gam_L} <S, dS'> + sum_i e^{gam_L-gam_i} k_i.(Vn dS'^T)_i;   dg = reverse chunk-local cumsum(dgam)
//      with dq, dk summed over the value heads of a GVA group in registers (deterministic, no atomics).
//      Replaces chunk_bwd_dqkwg + prepare_wy_repr_bwd_da + prepare_wy_repr_bwd_full + the reverse cumsum
//      (examples/flash_gated_delta_rule.py:962-1021).
//
// Operands the gradients are sensitive to travel as bf16 hi + bf16 residual and are multiplied in two or three
// tcgen05.mma passes; q, k, dO enter as the exact bf16 inputs; accumulation is fp32 in TMEM.
#include <algorithm>
#include "gdn_common.cuh"
#include "fla_b200_internal.h"
#include "kernel_timer.h"
#include "aux_stream.h"
#include "tensor_map.h"

namespace fla {

struct GdnBwdParams {
  const bf16* q; const bf16* k; const bf16* v; const bf16* dO;
  const void* beta;
  const float* q_rstd; const float* k_rstd;   // [tokens, HK] or null: q, k are normalised rows, dq / dk go through the normalisation
  const float* gam; const bf16* X;
  const bf16* s_img; const bf16* vn_img; const bf16* p_img;
  bf16* ds_img;        // [chunks, HV, V/32, 2, 128x32]  state gradient entering each chunk (hi, lo)
  bf16* dz_img;        // [chunks, HV, V/32, 192x32: rows 0-63 dO, rows 64-127 dZ rounded to bf16, rows 128-191 the residual of dZ]
  float* bz;           // [V/32, tokens, HV] partial sums of dZ * V over the 32-column slices of V
  const float* dht; float* dh0;
  const bf16* seg_m;   // [segments, HV, 128x128 (value, residual)]  the forward's transition matrices (split chains only)
  float* seg_dh;       // [segments, HV, V/128, 128, 128]
  int seg_len;         // chunks per segment
  int* counter;        // tiles the par kernel has handed out beyond its first wave; the scan in front of it sets it to zero
  void* dq; void* dk; void* dv; void* dg; void* dbeta;
  const int32_t* cu_seqlens; const int32_t* chunk_offsets;
  int64_t q_st, q_sh, k_st, k_sh, v_st, v_sh, do_st, do_sh, beta_st;
  int64_t dq_st, dq_sh, dk_st, dk_sh, dv_st, dv_sh;
  int64_t total_tokens;
  int N, T, HK, HV, beta_is_f32;
  int dq_f32, dk_f32, dv_f32, dg_f32, dbeta_f32;   // gradients leave in the dtypes of their inputs: f32, else bf16
  int V, nvb;          // value head dim (128 or 256) and its number of 64-column blocks
  int n0, n1;          // sequences of this launch (the backward may be launched as two halves of the batch)
  float scale;
  int* status;
};

}  // namespace fla
#include "gdn_scan_bwd.cuh"
namespace fla {

constexpr int64_t kSImg = 16384;   // bf16 elements of the state images per (chunk, head, 64-column block of V): (hi, lo) x 128x64
constexpr int64_t kVnImg = 8192;   // v_new images per (chunk, head, block): (hi, lo) x 64x64
constexpr int64_t kDzImg = kDzHalf;   // per (chunk, head, block): 64x64 dO, 64x64 dZ and the residual of dZ

// ============================================================================================= par
constexpr uint32_t rOffQK = 0, rQKPanel = 16384;
// Two stages, each the operands of 32 value channels (un-swizzled strips of 512 bytes, sm100.cuh, whose 32 rows are value channels: the
// reduction dim of these products).  [0 | residual of dZ^T]: the zeros are written once.  v_new^T and S strips, value / residual, are interleaved so
// that [Vn_lo | S_hi] and [Vn_hi | S_lo] are each one contiguous B operand of 24 strips.  As an A operand with valid rows 64..127 the view of
// v_new^T starts 4 KB earlier, inside the dZ^T strips or the S strips (any finite contents do).
constexpr uint32_t rOffStage = 32768, kStageStride = 57344;
constexpr uint32_t sOffAL = 0, sOffAH = 8192, sOffVNL = 16384, sOffSH = 20480, sOffVNH = 28672, sOffSL = 32768, sOffDSH = 40960, sOffDSL = 49152;
constexpr uint32_t kStageBytes = 12288 + 8192 + 16384 + 16384;      // loaded per stage
// [dP ; dAt] value / residual (128 rows x 64), behind 16 KB of zeros: read along the reduction over i, the zeros are the rows 0..63 of
// [0 ; dP^T | dAt^T], whose product then adds to the k-side rows alone and shares the accumulator of [dP; dAt] K.
constexpr uint32_t rOffZero = rOffStage + 2 * kStageStride, rOffPAH = rOffZero + 16384, rOffPAL = rOffPAH + 16384;
constexpr uint32_t kParSmem = rOffPAL + 16384;
constexpr uint32_t rColQK = 0, rColDV = 64, rColTA = 128, rColTB = 256, rColT2 = 384;
constexpr int kParWorkers = 512, kParThreads = kParWorkers + 128;      // + products, loader, two tail warps

// barrier `id` over `threads` threads that tells all of them whether all are fine
template <int kId, int kThreads>
__device__ __forceinline__ bool par_sync_and(bool ok) {
  uint32_t r;
  asm volatile(
      "{\n"
      " .reg .pred p, q;\n"
      " setp.ne.u32 q, %1, 0;\n"
      " bar.red.and.pred p, %2, %3, q;\n"
      " selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(r)
      : "r"(uint32_t(ok)), "n"(kId), "n"(kThreads)
      : "memory");
  return r != 0;
}

// Four neighbouring lanes hold four 16-byte pieces each: afterwards lane l has piece l % 4 of each of the four lanes.
__device__ __forceinline__ void transpose4x4(uint4 (&v)[4], int lane) {
  auto trade = [&](uint4& keep0, uint4& keep1, int bit) {      // the lane with the bit set keeps its second piece, the other its first
    const bool up = (lane & bit) != 0;
    const uint4 out = up ? keep0 : keep1;
    uint4 in;
    in.x = __shfl_xor_sync(0xffffffffu, out.x, bit); in.y = __shfl_xor_sync(0xffffffffu, out.y, bit);
    in.z = __shfl_xor_sync(0xffffffffu, out.z, bit); in.w = __shfl_xor_sync(0xffffffffu, out.w, bit);
    if (up) keep0 = in;
    else keep1 = in;
  };
  trade(v[0], v[1], 1);
  trade(v[2], v[3], 1);
  trade(v[0], v[2], 2);
  trade(v[1], v[3], 2);
}

struct ParItem {      // one value head of one (chunk, q/k head) tile
  int tile, h;        // h < 0: no more items
  int tok0, rows;
};

// One CTA per SM walks over (chunk, q/k head) tiles, handed out by a counter (next to the other half of the batch's scan, below, the CTAs do
// not start together); an item is one value head of a tile.
//     loader     operands of 32 value channels at a time into two stages; q, k of the next tile once the last item's readers are through
//     products   per stage [dO; dZ] . [Vn | S]^T and Vn . dS'^T; then, once [dP; dAt] is there, T2 = [dP; dAt] K + [0; dP^T | dAt^T] [Q; K]
//     workers    (sixteen warps) <S, dS'> of each stage; epilogue 1: score gradients -> [dP; dAt], first parts of dq / dk from the accumulators,
//                which the next item's products may overwrite from there on; epilogue 2: T2, row dots; after the last head dq, dk
//     tail       (two warps) gates and beta of the next item, dg and dbeta of the item before
// Loads, the products of the next item and the epilogues of this one overlap.  What bounded the one-tile-per-CTA form with eight warps (41,000
// cycles for a tile of two heads, of which shared memory needs 16,000 and HBM 19,000) was that they did not: load, products, load,
// products, epilogue, products, epilogue ran one after the other, each waited for by everything else.  Now about 20,000 - 25,000:
// 32,768 tokens, 16 / 32 heads 1.26 -> 0.86 ms, 8,191 packed tokens with 4 / 8 heads 112 -> 87 us.
// The products are issued from a one-thread branch: by the whole converged warp they go out faster than the tensor core takes them and the
// loads and epilogues that run beside them slow everything down (95 us for the packed batch).
// NVB: 64-column blocks of V per head (2 or 4), a compile-time trip count that keeps the stage loop unrolled.
template <int NVB>
__global__ void __launch_bounds__(kParThreads, 1) gdn_bwd_par_kernel(GdnBwdParams p, int chunks, const __grid_constant__ CUtensorMap tm_q,
                                                                     const __grid_constant__ CUtensorMap tm_k) {
  constexpr int NS = 2 * NVB;      // stages per item
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  // double-buffered by item parity
  __shared__ __align__(16) float gam_s2[2][kC], beta_s2[2][kC];
  __shared__ float red2[2][5][4][kC];      // q.dq, k.dk, rkG, rkB, ma : [32-column group of the row][row]
  __shared__ float sds_s2[2][kParWorkers / 32], ndot_s[4][2 * kC], fin_s[2][2];
  __shared__ ParItem item_s[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ __align__(8) uint64_t item_bar[2], qk_bar, full_bar[2];     // from the loader
  __shared__ __align__(8) uint64_t empty_bar[2];                         // stage read by the products and by every worker warp
  __shared__ __align__(8) uint64_t scal_bar[2], red_bar[2];              // tail: gam_s, beta_s there; worker warps: red2 there
  __shared__ __align__(8) uint64_t p1_bar, t2_bar;                       // products: all stages of an item, T2
  __shared__ __align__(8) uint64_t pa_bar, acc_bar, free_bar;            // worker warps: [dP; dAt] there, accumulators read, q and k read

  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  pdl_trigger();
  pdl_wait();
  const int G = p.HV / p.HK;
  // chunks of this launch: fixed lengths count from the first chunk of sequence n0, a packed batch's half is cut out here
  int chunk0 = 0;
  if (p.cu_seqlens) {
    chunk0 = p.chunk_offsets[p.n0];
    chunks = p.chunk_offsets[p.n1] - chunk0;
  }
  const int tiles = chunks * p.HK;
  const int flat0 = p.cu_seqlens ? chunk0 : p.n0 * ((p.T + kC - 1) / kC);      // flat index of the launch's first chunk

  if (warp == 0) {
    tmem_alloc(&tmem_base_s, 512);
    tmem_relinquish();
  }
  if (tid == 0) {
    for (uint64_t* b : {&item_bar[0], &item_bar[1], &qk_bar, &full_bar[0], &full_bar[1], &p1_bar, &t2_bar}) mbar_init(b, 1);
    for (uint64_t* b : {&pa_bar, &acc_bar, &free_bar, &red_bar[0], &red_bar[1]}) mbar_init(b, kParWorkers / 32);
    for (uint64_t* b : {&scal_bar[0], &scal_bar[1]}) mbar_init(b, 2);
    for (uint64_t* b : {&empty_bar[0], &empty_bar[1]}) mbar_init(b, kParWorkers / 32 + 1);
    mbar_init_fence();
  }
  if (tid < kParWorkers) {
    const uint4 z = make_uint4(0, 0, 0, 0);
    if (tid < 256) *reinterpret_cast<uint4*>(smem + rOffStage + sOffAL + tid * 16) = z;
    else *reinterpret_cast<uint4*>(smem + rOffStage + kStageStride + sOffAL + (tid - 256) * 16) = z;
    *reinterpret_cast<uint4*>(smem + rOffZero + tid * 16) = z;
    *reinterpret_cast<uint4*>(smem + rOffZero + 8192 + tid * 16) = z;
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = tmem_base_s;
  const uint32_t sb = smem_u32(smem);
  auto wait = [&](uint64_t* bar, uint32_t& phase) {
    const bool r = mbar_wait(bar, phase, p.status, FLA_ERR_TIMEOUT);
    phase ^= 1;
    return r;
  };
  // barriers that exist twice serve alternate items: their users may be an item apart
  auto wait_item = [&](uint64_t* bars, int n) { return mbar_wait(bars + (n & 1), (n >> 1) & 1, p.status, FLA_ERR_TIMEOUT); };
  auto signal = [&](uint64_t* bar) {      // my warp is done with what the barrier stands for
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
  };

  if (warp == kParWorkers / 32 + 1) {      // ---------------------------------------------------------------- loader
    auto first_stage = [&](int tile, int h) { return (int64_t(flat0 + tile / p.HK) * p.HV + (tile % p.HK) * G + h) * NS; };
    // A stage is seven copies, one lane each: a single thread took 1,000 cycles to issue them.  (Asking the stages after next into L2 as
    // well changed nothing at 4,096 to 32,768 tokens.)
    //               dO dZ   dZ_lo  Vn_hi  Vn_lo  S_hi   S_lo   dS
    const int img = lane < 2 ? 0 : lane < 4 ? 1 : lane < 6 ? 2 : 3;
    const int64_t stride = img == 0 ? 6144 : img == 1 ? 4096 : 8192;      // bf16 elements per stage
    const uint32_t dst = lane == 0 ? sOffAH : lane == 1 ? sOffAL + 4096 : lane == 2 ? sOffVNH : lane == 3 ? sOffVNL : lane == 4 ? sOffSH : lane == 5 ? sOffSL : sOffDSH;
    const uint32_t bytes = lane == 0 ? 8192 : lane < 4 ? 4096 : lane < 6 ? 8192 : 16384;
    const bf16* src = (img == 0 ? p.dz_img : img == 1 ? p.vn_img : img == 2 ? p.s_img : p.ds_img) + (lane == 1 ? 4096 : lane == 3 ? 2048 : lane == 5 ? 4096 : 0);
    auto position = [&](int tile) { return chunk_pos(p.cu_seqlens, p.chunk_offsets, p.N, p.T, p.n0, chunk0 + tile / p.HK); };

    uint32_t ph_empty[2] = {0, 0}, ph_free = 0;
    int tile = blockIdx.x, h = 0;
    int tok0 = 0, rows = 0;
    int64_t b0 = 0;
    if (tile < tiles) {
      const ChunkPos pos = position(tile);
      tok0 = pos.sq.bos + pos.c * kC;
      rows = min(kC, pos.sq.len - pos.c * kC);
      b0 = first_stage(tile, 0);
    }
    bool ok = true;
    for (int n = 0; ok; ++n) {
      if (lane == 0) {
        item_s[n & 1] = ParItem{tile, tile < tiles ? h : -1, tok0, rows};
        mbar_arrive(&item_bar[n & 1]);
      }
      if (tile >= tiles) break;
      int next = tile, hn = h + 1, tok0n = tok0, rowsn = rows;      // the item that follows
      int64_t bn = b0 + NS;
#pragma unroll
      for (int st = 0; st < NS; ++st) {
        const int s = st & 1;
        if (n > 0 || st >= 2) ok = ok && wait(&empty_bar[s], ph_empty[s]);
        ok = __shfl_sync(0xffffffffu, int(ok), 0) != 0;
        if (!ok) break;
        if (lane == 0) mbar_arrive_expect_tx(&full_bar[s], kStageBytes);
        __syncwarp();
        if (lane < 7) bulk_load(sb + rOffStage + s * kStageStride + dst, src + (b0 + st) * stride, bytes, &full_bar[s]);
        if (st == 1 && hn == G) {      // (while the stages are being read)
          hn = 0;
          if (lane == 0) next = int(gridDim.x) + atomicAdd(p.counter, 1);
          next = __shfl_sync(0xffffffffu, next, 0);
          if (next < tiles) {
            const ChunkPos pos = position(next);
            tok0n = pos.sq.bos + pos.c * kC;
            rowsn = min(kC, pos.sq.len - pos.c * kC);
            bn = first_stage(next, 0);
          }
        }
      }
      if (!ok) break;
      // q, k rows of the chunk (shared by the value heads of the group): four 64 x 64 tiles, for the score product at the end of the stages.  Rows
      // past the end of the sequence hold whatever follows in memory; every product with them meets a zero row or column of dO, dZ, v_new or
      // the masked score gradients, and those rows are never stored.
      if (h == 0) {
        if (n > 0) ok = wait(&free_bar, ph_free);
        if (lane == 0 && ok) {
          const int hk = tile % p.HK;
          mbar_arrive_expect_tx(&qk_bar, 32768);
          tma_load_tile(sb + rOffQK, &tm_q, 0, hk, tok0, &qk_bar);
          tma_load_tile(sb + rOffQK + 8192, &tm_k, 0, hk, tok0, &qk_bar);
          tma_load_tile(sb + rOffQK + rQKPanel, &tm_q, 64, hk, tok0, &qk_bar);
          tma_load_tile(sb + rOffQK + rQKPanel + 8192, &tm_k, 64, hk, tok0, &qk_bar);
        }
        __syncwarp();
      }
      tile = next, h = hn, tok0 = tok0n, rows = rowsn, b0 = bn;
    }
  } else if (warp == kParWorkers / 32) {      // ------------------------------------------------------------ products
    if (lane == 0) {
      const Operand opQK{sb + rOffQK, rQKPanel, 0};                      // [q; k], reduction over key dims
      const Operand opKb{sb + rOffQK + 8192, rQKPanel, 0};               // k as B, N = 64 tokens
      const Operand opKn{sb + rOffQK + 8192, rQKPanel, 1};               // k as B, N = 128 key dims, reduction over tokens
      const Operand opQKn{sb + rOffQK, rQKPanel, 1};                     // [q; k] as B, N = 128 key dims, reduction over 128 rows
      const Operand opPAH{sb + rOffPAH, 16384, 0}, opPAL{sb + rOffPAL, 16384, 0};                                            // [dP; dAt], reduction over j
      const Operand opPATh{sb + rOffZero, rOffPAH - rOffZero, 1}, opPATl{sb + rOffZero, rOffPAL - rOffZero, 1};              // [0; its transpose]
      uint32_t ph_full[2] = {0, 0}, ph_qk = 0, ph_pa = 0, ph_acc = 0;
      for (int n = 0;; ++n) {
        if (!wait_item(item_bar, n)) break;
        const int h = item_s[n & 1].h;
        if (h < 0) break;
        if (n > 0 && !wait(&acc_bar, ph_acc)) break;
        tc_fence_after();
        bool ok = true;
#pragma unroll
        for (int st = 0; st < NS; ++st) {
          const int s = st & 1;
          ok = ok && wait(&full_bar[s], ph_full[s]);
          if (!ok) break;
          const uint32_t base = sb + rOffStage + s * kStageStride;
          const Operand opAH{base + sOffAH, 512, 2};                                       // [dO; dZ]: M = 128 tokens = 16 strips
          const Operand opAL{base + sOffAL, 512, 2};                                       // [0; residual of dZ]: enters dA = -tril(dZ Vn^T) only
          const Operand opVNbL{base + sOffVNL, 512, 2}, opVNbH{base + sOffVNH, 512, 2};    // Vn as B (N = 64 tokens), S (N = 128 key dims) behind it
          const Operand opVNaH{base + sOffVNH - 4096, 512, 2}, opVNaL{base + sOffVNL - 4096, 512, 2};   // Vn as A: rows 64..127 are valid
          const Operand opDSH{base + sOffDSH, 512, 2}, opDSL{base + sOffDSL, 512, 2};
          const bool acc = st > 0;
          // [dO; dZ] . [Vn_lo | S_hi]^T and [dO; dZ] . [Vn_hi | S_lo]^T as N = 192 products: the A operand is read once for both
          static_assert(sOffVNL + 4096 == sOffSH && sOffVNH + 4096 == sOffSL && rColDV + 64 == rColTA, "the N = 192 products need these adjacent");
          mma_tile(tbase + rColDV, opAH, opVNbL, 128, 192, 2, acc);
          mma_tile(tbase + rColDV, opAH, opVNbH, 128, 192, 2, true);
          mma_tile(tbase + rColDV, opAL, opVNbH, 128, 64, 2, true);
          mma_tile(tbase + rColTB, opVNaH, opDSH, 128, 128, 2, acc);
          mma_tile(tbase + rColTB, opVNaH, opDSL, 128, 128, 2, true);
          mma_tile(tbase + rColTB, opVNaL, opDSH, 128, 128, 2, true);
          mma_commit(&empty_bar[s]);
        }
        if (ok && h == 0) {      // the score tiles of the chunk, kept for all heads of the group
          ok = wait(&qk_bar, ph_qk);
          if (ok) mma_tile(tbase + rColQK, opQK, opKb, 128, 64, 8, false);
        }
        if (!ok) break;
        mma_commit(&p1_bar);
        if (!wait(&pa_bar, ph_pa)) break;
        tc_fence_after();
        mma_tile(tbase + rColT2, opPAH, opKn, 128, 128, 4, false);
        mma_tile(tbase + rColT2, opPAL, opKn, 128, 128, 4, true);
        mma_tile(tbase + rColT2, opPATh, opQKn, 128, 128, 8, true);
        mma_tile(tbase + rColT2, opPATl, opQKn, 128, 128, 8, true);
        mma_commit(&t2_bar);
      }
    }
  } else if (warp > kParWorkers / 32) {      // ------------------------------------------------------------------ tail
    const int i = tid - (kParThreads - 64), w = i >> 5;      // my token
    bool ok = true;
    int rows0 = 0;          // of the item before: row count (0: none), where its dg / dbeta element goes, its scalars
    int64_t gidx0 = 0;
    float gv0 = 0.f, bv0 = 0.f, bz0 = 0.f;
    for (int n = 0;; ++n) {
      ok = ok && wait_item(item_bar, n);
      const ParItem it = ok ? item_s[n & 1] : ParItem{0, 0, 0, 1};
      const bool more = it.h >= 0;
      const int hv = (it.tile % p.HK) * G + it.h;
      const int64_t gidx = (int64_t(it.tok0) + min(i, it.rows - 1)) * p.HV + hv;
      float gv = 0.f, bv = 0.f, bz = 0.f;
      if (more) {
        gv = p.gam[gidx] * kLog2e;
        if (i < it.rows) bv = ld_scalar(p.beta, (int64_t(it.tok0) + i) * p.beta_st + hv, p.beta_is_f32);
#pragma unroll
        for (int s = 0; s < 2 * NVB; ++s) bz += p.bz[s * p.total_tokens * p.HV + gidx];
        gam_s2[n & 1][i] = gv;
        beta_s2[n & 1][i] = bv;
        signal(&scal_bar[n & 1]);
      }
      // dg / dbeta rows of the item before.  dg = reverse chunk-local cumulative sum of dgam; the last row additionally carries
      // e^{gam_L} <S, dS'> + sum_i e^{gam_L - gam_i} k_i.(Vn dS'^T)_i, which therefore reaches every row.
      if (n > 0) ok = ok && wait_item(red_bar, n - 1);
      float suf = 0.f, tot3 = 0.f, tot = 0.f, gl = 0.f;
      const bool live = i < rows0;
      if (rows0) {
        float (*red)[4][kC] = red2[(n - 1) & 1];
        auto sum4 = [&](int r) { return (red[r][0][i] + red[r][1][i]) + (red[r][2][i] + red[r][3][i]); };
        const float qdq = sum4(0), kdk = sum4(1), g_ = sum4(2), b_ = sum4(3), ma = sum4(4), egi = exp2_fast(gv0);
        gl = gam_s2[(n - 1) & 1][rows0 - 1];
#pragma unroll
        for (int j = 0; j < kParWorkers / 32; ++j) tot += sds_s2[(n - 1) & 1][j];
        if (live) {
          suf = qdq - kdk + 2.f * bv0 * ma - 2.f * bv0 * egi * g_;
          tot3 = exp2_fast(gl - gv0) * b_;
          const float db = bz0 - egi * g_ + ma;
          if (p.dbeta_f32) static_cast<float*>(p.dbeta)[gidx0] = db;
          else static_cast<bf16*>(p.dbeta)[gidx0] = __float2bfloat16_rn(db);
        }
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float dn = __shfl_down_sync(0xffffffffu, suf, o);
        if (lane + o < 32) suf += dn;
        tot3 += __shfl_xor_sync(0xffffffffu, tot3, o);
      }
      if (lane == 0) {
        fin_s[0][w] = suf;      // total of this warp's 32 rows (suffix sum at its first row)
        fin_s[1][w] = tot3;
      }
      ok = par_sync_and<2, 64>(ok);
      if (live && ok) {
        if (w == 0) suf += fin_s[0][1];
        const float dgv = suf + exp2_fast(gl) * tot + fin_s[1][0] + fin_s[1][1];
        if (p.dg_f32) static_cast<float*>(p.dg)[gidx0] = dgv;
        else static_cast<bf16*>(p.dg)[gidx0] = __float2bfloat16_rn(dgv);
      }
      if (!ok || !more) break;
      par_sync_and<2, 64>(true);      // fin_s is free again
      rows0 = it.rows, gidx0 = gidx, gv0 = gv, bv0 = bv, bz0 = bz;
    }
  } else {      // ------------------------------------------------------------------------------------------ workers
    const int quad = warp & 3, cg = warp >> 2;  // my 32 accumulator rows, my 32 key-dim columns
    const int row = quad * 32 + lane;           // accumulator row == TMEM lane
    const bool kside = quad >= 2;
    const int tok = row & 63;
    const uint32_t trow = tmem_addr(tbase, quad * 32, 0);
    const uint8_t* qk = smem + rOffQK + (cg >> 1) * rQKPanel;      // the panel of my columns
    auto qk8 = [&](int ch, float* f) {      // eight elements of my row of [q; k]
      unpack_bf16x8(*reinterpret_cast<const uint4*>(qk + panel_chunk_off(row, (cg & 1) * 4 + ch)), f);
    };
    uint32_t ph_full[2] = {0, 0}, ph_qk = 0, ph = 0;
    bool ok = true;
    float acc[32];      // running dq (q-side rows) or dk (k-side rows), my 32 key-dim columns
#pragma unroll
    for (int i = 0; i < 32; ++i) acc[i] = 0.f;
    float xsum = 0.f;   // their dot product with q or k
    // My part of <S, dS'> of a stage, elementwise on the raw images.  Values and residuals: the terms have either sign, so the sum is no
    // larger than its rounding noise would be with the values alone (ragged chunks, where this term dominates dg, then miss by 10x).
    float sds = 0.f;
    auto stage_dot = [&](int s) {
      ok = ok && wait(&full_bar[s], ph_full[s]);
      const uint8_t* base = smem + rOffStage + s * kStageStride + tid * 16;
      const uint4 r1 = *reinterpret_cast<const uint4*>(base + sOffSH), r2 = *reinterpret_cast<const uint4*>(base + sOffSL);
      const uint4 r3 = *reinterpret_cast<const uint4*>(base + sOffDSH), r4 = *reinterpret_cast<const uint4*>(base + sOffDSL);
      float s1[8], s2[8], d1[8], d2[8];
      unpack_bf16x8(r1, s1);
      unpack_bf16x8(r2, s2);
      unpack_bf16x8(r3, d1);
      unpack_bf16x8(r4, d2);
#pragma unroll
      for (int j = 0; j < 8; ++j) sds += (s1[j] + s2[j]) * (d1[j] + d2[j]);
      signal(&empty_bar[s]);
    };
    ParItem it, next;
    // An item's first two stages are read while the products of the one before are waited for.  A wait that runs out makes this thread
    // skip the rest of its waits; all leave together at the barrier behind the stages.
    auto take = [&](int n) {
      ok = ok && wait_item(item_bar, n);
      next = ok ? item_s[n & 1] : ParItem{0, 0, 0, 1};
      sds = 0.f;
      if (next.h >= 0) {
        stage_dot(0);
        stage_dot(1);
      }
    };
    take(0);
    for (int n = 0;; ++n) {
      it = next;
      if (it.h < 0) {
        par_sync_and<1, kParWorkers>(true);
        break;
      }
#pragma unroll
      for (int st = 2; st < NS; ++st) stage_dot(st & 1);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sds += __shfl_xor_sync(0xffffffffu, sds, o);
      const int hk = it.tile % p.HK, rows = it.rows;
      const int64_t tok0 = it.tok0;
      const float *gam_s = gam_s2[n & 1], *beta_s = beta_s2[n & 1];
      float (*red)[4][kC] = red2[n & 1];
      ok = ok && wait_item(scal_bar, n);
      if (lane == 0) sds_s2[n & 1][warp] = sds;
      if (it.h == 0) ok = ok && wait(&qk_bar, ph_qk);
      ok = par_sync_and<1, kParWorkers>(ok);
      if (!ok) break;

      // ---- epilogue 1: score-tile gradients -> [dP; dAt] operand, first parts of this head's dq / dk rows
      ok = mbar_wait(&p1_bar, ph, p.status, FLA_ERR_TIMEOUT);
      tc_fence_after();
      const float gam_i = gam_s[tok], beta_i = beta_s[tok], eg = exp2_fast(gam_i);
      {
        float sc[16], dvv[16];
        tmem_ld16(trow + rColQK + cg * 16, sc);
        tmem_ld16(trow + rColDV + cg * 16, dvv);
        float ma = 0.f;
        tmem_ld_wait();
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {
          float t[8];
          gather8(gam_s + cg * 16 + ch * 8, t);
          if (!kside) {
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) {
              const float e = p.scale * exp2_fast(fminf(gam_i - t[jj], 0.f));
              dvv[ch * 8 + jj] *= (cg * 16 + ch * 8 + jj <= tok) ? e : 0.f;
            }
          } else {
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) {
              const float e = exp2_fast(fminf(gam_i - t[jj], 0.f));
              const float dA = (cg * 16 + ch * 8 + jj < tok) ? -dvv[ch * 8 + jj] * e : 0.f;
              ma += dA * sc[ch * 8 + jj];
              dvv[ch * 8 + jj] = dA * beta_i;
            }
          }
          uint4 hi, lo;
          split8(dvv + ch * 8, hi, lo);
          const uint32_t off = panel_chunk_off(row, cg * 2 + ch);
          *reinterpret_cast<uint4*>(smem + rOffPAH + off) = hi;
          *reinterpret_cast<uint4*>(smem + rOffPAL + off) = lo;
        }
        if (kside) red[4][cg][tok] = ma;
      }
      fence_async_smem();
      tc_fence_before();
      signal(&pa_bar);
      float xdx = 0.f;      // q.dq (q-side) or k.dk (k-side) over my columns, this head's part
      if (!kside) {
        const float f = p.scale * eg;
#pragma unroll
        for (int c2 = 0; c2 < 2; ++c2) {
          float x[16];
          tmem_ld16(trow + rColTA + cg * 32 + c2 * 16, x);
          float qv[16];
          qk8(c2 * 2, qv);
          qk8(c2 * 2 + 1, qv + 8);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            x[i] *= f;
            xdx += qv[i] * x[i];
            acc[c2 * 16 + i] += x[i];
          }
        }
      } else {
        const float f1 = -beta_i * eg, f2 = exp2_fast(gam_s[rows - 1] - gam_i);
        float rkG = 0.f, rkB = 0.f;
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
          float x[8], y[8], kv[8];
          tmem_ld8(trow + rColTA + cg * 32 + ch * 8, x);
          tmem_ld8(trow + rColTB + cg * 32 + ch * 8, y);
          qk8(ch, kv);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            rkG += kv[i] * x[i];
            rkB += kv[i] * y[i];
            acc[ch * 8 + i] += f1 * x[i] + f2 * y[i];
          }
        }
        red[2][cg][tok] = rkG;
        red[3][cg][tok] = rkB;
        xdx = f1 * rkG + f2 * rkB;
      }
      tc_fence_before();
      signal(&acc_bar);
      take(n + 1);

      // ---- epilogue 2: finish the rows, row dots for dg / dbeta
      const bool last = it.h + 1 == G;
      float rs = 0.f;
      if (last && p.q_rstd) rs = (kside ? p.k_rstd : p.q_rstd)[(tok0 + min(tok, rows - 1)) * p.HK + hk];
      ok = ok && mbar_wait(&t2_bar, ph, p.status, FLA_ERR_TIMEOUT);
      tc_fence_after();
#pragma unroll
      for (int c2 = 0; c2 < 2; ++c2) {
        float x[16], v[16];
        tmem_ld16(trow + rColT2 + cg * 32 + c2 * 16, x);
        qk8(c2 * 2, v);
        qk8(c2 * 2 + 1, v + 8);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          xdx += v[i] * x[i];
          acc[c2 * 16 + i] += x[i];
        }
      }
      red[kside ? 1 : 0][cg][tok] = xdx;
      tc_fence_before();
      xsum += xdx;
      if (last && p.q_rstd) ndot_s[cg][row] = xsum;
      signal(&red_bar[n & 1]);
      ph ^= 1;
      if (!last) continue;

      if (p.q_rstd) {   // the rows are complete: through the normalisation, rstd (dx - x (x . dx))
        ok = par_sync_and<1, kParWorkers>(ok);
        const float t = (ndot_s[0][row] + ndot_s[1][row]) + (ndot_s[2][row] + ndot_s[3][row]);
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
          float f[8];
          qk8(ch, f);
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[ch * 8 + j] = (acc[ch * 8 + j] - t * f[j]) * rs;
        }
      }
      signal(&free_bar);
      {
        void* base = kside ? p.dk : p.dq;
        const int64_t st_ = kside ? p.dk_st : p.dq_st;
        const int64_t off = tok0 * st_ + hk * (kside ? p.dk_sh : p.dq_sh) + cg * 32;
        if (kside ? p.dk_f32 : p.dq_f32) {
          float* dst = static_cast<float*>(base) + off + tok * st_;
          if (tok < rows) {
#pragma unroll
            for (int i = 0; i < 32; i += 4) *reinterpret_cast<float4*>(dst + i) = make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
          }
        } else {      // four lanes trade pieces so that they store 64 contiguous bytes of one row after the other
          uint4 v[4];
#pragma unroll
          for (int ch = 0; ch < 4; ++ch) v[ch] = pack8(acc + ch * 8);
          transpose4x4(v, lane);
          bf16* dst = static_cast<bf16*>(base) + off + (tok & ~3) * st_ + (lane & 3) * 8;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if ((tok & ~3) + j < rows) *reinterpret_cast<uint4*>(dst + j * st_) = v[j];
        }
      }
      xsum = 0.f;
#pragma unroll
      for (int i = 0; i < 32; ++i) acc[i] = 0.f;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tbase, 512);
}

}  // namespace fla

using namespace fla;

static uint64_t bwd_ws_layout(int64_t total_chunks, int64_t HV, int64_t nvb, int64_t tokens, const SegPlan& plan, uint64_t* off_ds,
                              uint64_t* off_dz, uint64_t* off_bz, uint64_t* off_seg) {
  uint64_t o = 256;  // status block
  *off_ds = o; o += align_up(uint64_t(total_chunks) * HV * nvb * kSImg * 2, 256);
  *off_dz = o; o += align_up(uint64_t(total_chunks) * HV * nvb * kDzImg * 2, 256);
  *off_bz = o; o += align_up(uint64_t(2 * nvb) * tokens * HV * 4, 256);
  *off_seg = o;
  if (plan.split) o += uint64_t(plan.count) * HV * (nvb / 2) * kSegHBytes;
  return o;
}

static int bwd_geometry(const fla_gdn_chunk_bwd_args* a, int64_t* total_chunks, int* N) {
  const fla_tensor_t& q = a->q;
  if (!q.data || q.ndim != 4 || !a->v.data || a->v.ndim != 4) return FLA_ERR_SHAPE;
  const int64_t B = q.shape[0], T = q.shape[1];
  *N = int(B);
  *total_chunks = B * ((T + kC - 1) / kC);
  if (a->cu_seqlens.data) {
    if (B != 1 || a->cu_seqlens.dtype != FLA_I32 || a->cu_seqlens.ndim != 1 || a->cu_seqlens.shape[0] < 2) return FLA_ERR_SHAPE;
    *N = int(a->cu_seqlens.shape[0] - 1);
    if (!a->chunk_offsets.data || a->chunk_offsets.dtype != FLA_I32 || a->chunk_offsets.shape[0] != *N + 1) return FLA_ERR_SHAPE;
    if (a->max_seqlen <= 0 || a->max_seqlen > T || a->total_chunks <= 0) return FLA_ERR_VALUE;
    *total_chunks = a->total_chunks;
  }
  return FLA_OK;
}

static SegPlan bwd_plan(const fla_gdn_chunk_bwd_args* a, int64_t total_chunks, int N) {
  SegPlan whole;
  whole.count = N;
  if (!a->seg_m.data) return whole;
  const bool packed = a->cu_seqlens.data != nullptr;
  return scan_plan(N, total_chunks, packed ? a->max_seqlen : a->q.shape[1], packed, a->v.shape[2], a->v.shape[3]);
}

extern "C" FLA_API int fla_b200_gdn_chunk_bwd_workspace_size(const fla_gdn_chunk_bwd_args* a, uint64_t* bytes) {
  if (!a || !bytes) return FLA_ERR_NULL;
  int64_t total_chunks; int N;
  int st = bwd_geometry(a, &total_chunks, &N);
  if (st) return st;
  uint64_t o1, o2, o3, o4;
  const int64_t V = a->v.shape[3];
  if (V != kV && V != 2 * kV) return FLA_ERR_SHAPE;
  *bytes = bwd_ws_layout(total_chunks, a->v.shape[2], V / kBV, a->q.shape[0] * a->q.shape[1], bwd_plan(a, total_chunks, N), &o1, &o2, &o3, &o4);
  return FLA_OK;
}

static int check_tok4(const fla_tensor_t& t, int64_t B, int64_t T, int64_t heads, int64_t dim, bool allow_f32) {
  if (!t.data) return FLA_ERR_NULL;
  if (t.ndim != 4 || t.shape[0] != B || t.shape[1] != T || t.shape[2] != heads || t.shape[3] != dim) return FLA_ERR_SHAPE;
  if (t.dtype != FLA_BF16 && !(allow_f32 && t.dtype == FLA_F32)) return FLA_ERR_DTYPE;
  const int64_t esz = t.dtype == FLA_F32 ? 4 : 2;
  if (t.stride[3] != 1 || (t.stride[2] * esz) % 16 || (t.stride[1] * esz) % 16 || !aligned16(t.data)) return FLA_ERR_LAYOUT;
  if (B > 1 && t.stride[0] != T * t.stride[1]) return FLA_ERR_LAYOUT;
  return FLA_OK;
}
static int check_tok3(const fla_tensor_t& t, int64_t B, int64_t T, int64_t heads, bool dense) {
  if (!t.data) return FLA_ERR_NULL;
  if (t.ndim != 3 || t.shape[0] != B || t.shape[1] != T || t.shape[2] != heads) return FLA_ERR_SHAPE;
  if (t.dtype != FLA_BF16 && t.dtype != FLA_F32) return FLA_ERR_DTYPE;
  if (t.stride[2] != 1 || (B > 1 && t.stride[0] != T * t.stride[1])) return FLA_ERR_LAYOUT;
  if (dense && t.stride[1] != heads) return FLA_ERR_LAYOUT;
  return FLA_OK;
}


static int gdn_chunk_bwd_impl(const fla_gdn_chunk_bwd_args* a, void* workspace, uint64_t workspace_bytes, void* stream,
                              bool allow_split) {
  if (!a) return FLA_ERR_NULL;
  int64_t total_chunks; int N;
  int st = bwd_geometry(a, &total_chunks, &N);
  if (st) return st;
  const int64_t B = a->q.shape[0], T = a->q.shape[1], HK = a->q.shape[2], HV = a->v.shape[2];
  if (HK <= 0 || HV <= 0 || HV % HK) return FLA_ERR_SHAPE;
  const int64_t V = a->v.shape[3], nvb = V / kBV;
  if (V != kV && V != 2 * kV) return FLA_ERR_SHAPE;
  if ((st = check_tok4(a->q, B, T, HK, kK, false))) return st;
  if ((st = check_tok4(a->k, B, T, HK, kK, false))) return st;
  if ((st = check_tok4(a->v, B, T, HV, V, false))) return st;
  if ((st = check_tok4(a->d_o, B, T, HV, V, false))) return st;
  if ((st = check_tok4(a->dq, B, T, HK, kK, true))) return st;
  if ((st = check_tok4(a->dk, B, T, HK, kK, true))) return st;
  if ((st = check_tok4(a->dv, B, T, HV, V, true))) return st;
  if ((st = check_tok3(a->beta, B, T, HV, false))) return st;
  if ((st = check_tok3(a->dg, B, T, HV, true))) return st;
  if ((st = check_tok3(a->dbeta, B, T, HV, true))) return st;
  const fla_tensor_t &gam = a->gam, &X = a->x_inv;
  if (!gam.data || !X.data || !a->s_img.data || !a->vn_img.data || !a->p_img.data) return FLA_ERR_NULL;
  if (gam.dtype != FLA_F32 || gam.ndim != 3 || gam.shape[0] != B || gam.shape[1] != T || gam.shape[2] != HV ||
      gam.stride[2] != 1 || gam.stride[1] != HV || (B > 1 && gam.stride[0] != T * HV))
    return FLA_ERR_SHAPE;
  if (X.dtype != FLA_BF16 || X.ndim != 1 || X.shape[0] != total_chunks * HV * 8192 || !aligned16(X.data))
    return FLA_ERR_SHAPE;
  if (a->p_img.dtype != FLA_BF16 || a->p_img.ndim != 1 || a->p_img.shape[0] != total_chunks * HV * kPImg || !aligned16(a->p_img.data))
    return FLA_ERR_SHAPE;
  if (a->s_img.dtype != FLA_BF16 || a->s_img.ndim != 1 || a->s_img.shape[0] != total_chunks * HV * nvb * kSImg || !aligned16(a->s_img.data))
    return FLA_ERR_SHAPE;
  if (a->vn_img.dtype != FLA_BF16 || a->vn_img.ndim != 1 || a->vn_img.shape[0] != total_chunks * HV * nvb * kVnImg || !aligned16(a->vn_img.data))
    return FLA_ERR_SHAPE;
  for (const fla_tensor_t* s : {&a->dht, &a->dh0}) {
    if (!s->data) continue;
    if (s->dtype != FLA_F32) return FLA_ERR_DTYPE;
    if (s->ndim != 4 || s->shape[0] != N || s->shape[1] != HV || s->shape[2] != kK || s->shape[3] != V) return FLA_ERR_SHAPE;
    if (s->stride[3] != 1 || s->stride[2] != V || s->stride[1] != kK * V || s->stride[0] != HV * kK * V || !aligned16(s->data))
      return FLA_ERR_LAYOUT;
  }
  if (a->q_rstd.data || a->k_rstd.data) {
    for (const fla_tensor_t* t : {&a->q_rstd, &a->k_rstd}) {
      if (!t->data) return FLA_ERR_NULL;
      if (t->dtype != FLA_F32) return FLA_ERR_DTYPE;
      if ((st = check_tok3(*t, B, T, HK, true))) return st;
    }
  }
  if (a->chunk_size != kC) return FLA_ERR_VALUE;
  uint64_t off_ds, off_dz, off_bz, off_seg;
  const SegPlan plan = bwd_plan(a, total_chunks, N);
  if (plan.split && (a->seg_m.dtype != FLA_BF16 || a->seg_m.ndim != 1 || uint64_t(a->seg_m.shape[0]) * 2 < uint64_t(plan.count) * HV * kSegMBytes ||
                     !aligned16(a->seg_m.data)))
    return FLA_ERR_SHAPE;
  const uint64_t need = bwd_ws_layout(total_chunks, HV, nvb, B * T, plan, &off_ds, &off_dz, &off_bz, &off_seg);
  if (!workspace || workspace_bytes < need || !aligned16(workspace)) return FLA_ERR_WORKSPACE;

  GdnBwdParams p{};
  p.q = static_cast<const bf16*>(a->q.data); p.k = static_cast<const bf16*>(a->k.data);
  p.v = static_cast<const bf16*>(a->v.data); p.dO = static_cast<const bf16*>(a->d_o.data);
  p.q_rstd = static_cast<const float*>(a->q_rstd.data); p.k_rstd = static_cast<const float*>(a->k_rstd.data);
  p.beta = a->beta.data; p.gam = static_cast<const float*>(gam.data); p.X = static_cast<const bf16*>(X.data);
  p.s_img = static_cast<const bf16*>(a->s_img.data); p.vn_img = static_cast<const bf16*>(a->vn_img.data);
  p.p_img = static_cast<const bf16*>(a->p_img.data);
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  p.status = reinterpret_cast<int*>(ws);
  p.counter = p.status + 16;      // both inside the workspace's 256-byte head
  p.ds_img = reinterpret_cast<bf16*>(ws + off_ds);
  p.dz_img = reinterpret_cast<bf16*>(ws + off_dz);
  p.bz = reinterpret_cast<float*>(ws + off_bz);
  p.seg_m = static_cast<const bf16*>(a->seg_m.data);
  p.seg_dh = reinterpret_cast<float*>(ws + off_seg);
  p.seg_len = plan.len;
  p.dht = static_cast<const float*>(a->dht.data); p.dh0 = static_cast<float*>(a->dh0.data);
  p.dq = a->dq.data; p.dk = a->dk.data; p.dv = a->dv.data; p.dg = a->dg.data; p.dbeta = a->dbeta.data;
  p.cu_seqlens = static_cast<const int32_t*>(a->cu_seqlens.data);
  p.chunk_offsets = static_cast<const int32_t*>(a->chunk_offsets.data);
  p.q_st = a->q.stride[1]; p.q_sh = a->q.stride[2]; p.k_st = a->k.stride[1]; p.k_sh = a->k.stride[2];
  p.v_st = a->v.stride[1]; p.v_sh = a->v.stride[2]; p.do_st = a->d_o.stride[1]; p.do_sh = a->d_o.stride[2];
  p.beta_st = a->beta.stride[1];
  p.dq_st = a->dq.stride[1]; p.dq_sh = a->dq.stride[2]; p.dk_st = a->dk.stride[1]; p.dk_sh = a->dk.stride[2];
  p.dv_st = a->dv.stride[1]; p.dv_sh = a->dv.stride[2];
  p.total_tokens = B * T; p.n1 = N;
  p.N = N; p.T = int(T); p.HK = int(HK); p.HV = int(HV); p.V = int(V); p.nvb = int(nvb);
  p.beta_is_f32 = a->beta.dtype == FLA_F32;
  p.dq_f32 = a->dq.dtype == FLA_F32; p.dk_f32 = a->dk.dtype == FLA_F32; p.dv_f32 = a->dv.dtype == FLA_F32;
  p.dg_f32 = a->dg.dtype == FLA_F32; p.dbeta_f32 = a->dbeta.dtype == FLA_F32;
  p.scale = a->scale;

  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  static std::atomic<bool> attr_done_dev[64] = {};   // per device ordinal; setting the attributes twice is harmless
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return FLA_ERR_CUDA;
  if (!attr_done_dev[dev]) {
    for (auto* scan : {gdn_scan_bwd_kernel<false, false>, gdn_scan_bwd_kernel<false, true>, gdn_scan_bwd_kernel<true, true>})
      if (cudaFuncSetAttribute(scan, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kScanBwdSmem) + 1024) != cudaSuccess) return FLA_ERR_CUDA;
    if (cudaFuncSetAttribute(gdn_bwd_par_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kParSmem) + 1024) != cudaSuccess) return FLA_ERR_CUDA;
    if (cudaFuncSetAttribute(gdn_bwd_par_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kParSmem) + 1024) != cudaSuccess) return FLA_ERR_CUDA;
    attr_done_dev[dev] = true;
  }
  CUtensorMap tm_q, tm_k, tm_v, tm_d;
  if (make_row_tile_map(&tm_q, p.q, kK, uint64_t(HK), uint64_t(B * T), uint64_t(p.q_sh), uint64_t(p.q_st)) ||
      make_row_tile_map(&tm_k, p.k, kK, uint64_t(HK), uint64_t(B * T), uint64_t(p.k_sh), uint64_t(p.k_st)) ||
      make_row_tile_map(&tm_v, p.v, uint64_t(V), uint64_t(HV), uint64_t(B * T), uint64_t(p.v_sh), uint64_t(p.v_st)) ||
      make_row_tile_map(&tm_d, p.dO, uint64_t(V), uint64_t(HV), uint64_t(B * T), uint64_t(p.do_sh), uint64_t(p.do_st)))
    return FLA_ERR_CUDA;
  // The reverse scan launches one CTA per (sequence, value head, 128 channels) and each needs a whole SM: when there are
  // more chains than SMs the last round leaves SMs idle for the length of a chain.  The batch is then launched as two
  // halves on two streams, so that the chunk-parallel kernel of the first half fills the SMs the second half's scan
  // leaves free.  Not while per-kernel timing is on (its events bracket single launches), not during stream capture, not
  // for the allocation-free entry (creating the second stream may allocate).
  AuxStream* aux = nullptr;
  if (allow_split && N >= 2 && !plan.split && int64_t(V / 128) * HV * N > sm_count(dev) && !kernel_timing_enabled()) aux = aux_stream_for(dev, cs);
  auto launch_scan = [&](const GdnBwdParams& pp, int64_t segments, cudaStream_t st) {
    const dim3 grid(unsigned(HV * (V / 128)), unsigned(segments));
    if (plan.split) {
      const cudaError_t e = launch_after(!aux, gdn_scan_bwd_kernel<true, true>, grid, kScanThreads, kScanBwdSmem + 1024, st, pp, tm_q, tm_k, tm_v, tm_d);
      if (e != cudaSuccess) return e;
    }
    return launch_after(!aux, plan.split ? gdn_scan_bwd_kernel<false, true> : gdn_scan_bwd_kernel<false, false>, grid, kScanThreads, kScanBwdSmem + 1024, st, pp, tm_q,
                      tm_k, tm_v, tm_d);
  };
  auto launch_par = [&](const GdnBwdParams& pp, int64_t chunks, cudaStream_t st) {
    return launch_after(!aux, nvb == 2 ? gdn_bwd_par_kernel<2> : gdn_bwd_par_kernel<4>, unsigned(std::min<int64_t>(chunks * HK, sm_count(dev))), kParThreads,
                      kParSmem + 1024, st, pp, int(chunks), tm_q, tm_k);
  };
  if (aux) {
    std::lock_guard<std::mutex> lk(aux->mu);   // the fork / join events are shared by the callers of this stream
    const int n1 = N / 2;
    GdnBwdParams p2 = p;
    p.n1 = p2.n0 = n1;
    p2.counter = p.counter + 16;
    bool okc = cudaEventRecord(aux->fork, cs) == cudaSuccess && cudaStreamWaitEvent(aux->s, aux->fork, 0) == cudaSuccess;
    if (!okc) return FLA_ERR_CUDA;
    bool launched = launch_scan(p, n1, cs) == cudaSuccess && launch_scan(p2, N - n1, aux->s) == cudaSuccess;
    // a packed batch's halves hold chunk counts the host does not have: the kernel looks up its own
    const int64_t nt = (T + kC - 1) / kC;
    launched = launched && launch_par(p, p.cu_seqlens ? total_chunks : n1 * nt, cs) == cudaSuccess &&
               launch_par(p2, p.cu_seqlens ? total_chunks : (N - n1) * nt, aux->s) == cudaSuccess;
    okc = cudaEventRecord(aux->join, aux->s) == cudaSuccess && cudaStreamWaitEvent(cs, aux->join, 0) == cudaSuccess;
    if (!okc) return FLA_ERR_CUDA;
    return launched ? FLA_OK : FLA_ERR_CUDA;
  }
  {
    KernelTimer kt("gdn_bwd_dhu", cs);
    if (launch_scan(p, plan.count, cs) != cudaSuccess) return FLA_ERR_CUDA;
  }
  {
    KernelTimer kt("gdn_bwd_par", cs);
    return cuda_status(launch_par(p, total_chunks, cs));
  }
}

extern "C" FLA_API int fla_b200_gdn_chunk_bwd(const fla_gdn_chunk_bwd_args* a, void* workspace, uint64_t workspace_bytes,
                                              void* stream) {
  return gdn_chunk_bwd_impl(a, workspace, workspace_bytes, stream, true);
}

// ----------------------------------------------------------------------------- allocation-free variant
// Some hosts of this library may not allocate device memory at the point where they call the backward:
// an inference / training runtime that sized one device arena at start-up and forbids any later
// cudaMalloc (an allocation can synchronise the whole device and stall the other streams of a serving
// process), a plugin running inside another framework's callback that owns the allocator, or a
// real-time loop with a fixed memory budget.  For them the scratch that fla_b200_gdn_chunk_bwd normally
// receives from the caller lives here instead, in one fixed array that is part of the library image:
// every GPU whose context loads libfla_b200.so carries these 32 MiB until the process exits.
constexpr uint64_t kStaticScratchBytes = 32ull << 20;
static __device__ __align__(256) unsigned char g_bwd_static_scratch[kStaticScratchBytes];

#include <mutex>
namespace {
std::mutex g_static_mu;
void* g_static_ptr[64] = {};   // device address of the array, per device ordinal
}  // namespace

extern "C" FLA_API int fla_b200_gdn_chunk_bwd_static_scratch_bytes(uint64_t* bytes) {
  if (!bytes) return FLA_ERR_NULL;
  *bytes = kStaticScratchBytes;
  return FLA_OK;
}

extern "C" FLA_API int fla_b200_gdn_chunk_bwd_noalloc(const fla_gdn_chunk_bwd_args* a, void* stream) {
  if (!a) return FLA_ERR_NULL;
  uint64_t need = 0;
  const int st = fla_b200_gdn_chunk_bwd_workspace_size(a, &need);
  if (st != FLA_OK) return st;
  if (need > kStaticScratchBytes) return FLA_ERR_TOO_LARGE;   // the problem does not fit the built-in scratch
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return FLA_ERR_CUDA;
  void* scratch = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_static_mu);
    if (!g_static_ptr[dev]) {
      // In host code the array's name is only a handle; the address the kernels can use has to be asked for,
      // once per device, while that device is current.
      void* ptr = nullptr;
      if (cudaGetSymbolAddress(&ptr, g_bwd_static_scratch) != cudaSuccess || !ptr) return FLA_ERR_CUDA;
      g_static_ptr[dev] = ptr;
    }
    scratch = g_static_ptr[dev];
  }
  // The regular entry point's first kernel clears the status word at the head of the scratch on `stream` and overwrites
  // every other byte it later reads, so nothing else of the previous call's contents matters.
  return gdn_chunk_bwd_impl(a, scratch, kStaticScratchBytes, stream, false);   // one stream: creating a second one may allocate
}

// The status word of the allocation-free entry lives at the head of the built-in array, which the caller cannot
// address; this copies it out after waiting for `stream` (the stream of the call being checked).
extern "C" FLA_API int fla_b200_gdn_chunk_bwd_noalloc_status(void* stream, int32_t* status_out) {
  if (!status_out) return FLA_ERR_NULL;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return FLA_ERR_CUDA;
  void* scratch = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_static_mu);
    scratch = g_static_ptr[dev];
  }
  if (!scratch) {   // no call on this device yet: nothing has run, nothing can have timed out
    *status_out = FLA_OK;
    return FLA_OK;
  }
  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  int32_t word = 0;
  if (cudaMemcpyAsync(&word, scratch, sizeof(word), cudaMemcpyDeviceToHost, cs) != cudaSuccess) return FLA_ERR_CUDA;
  if (cudaStreamSynchronize(cs) != cudaSuccess) return FLA_ERR_CUDA;
  *status_out = word;
  return FLA_OK;
}

