// Chunked Kimi-Delta-Attention backward (per-channel log gate, chunk = 64, K = V = 128).
//
// The reference ships only the intra-chunk piece of this backward (chunk_kda_bwd_intra,
// torch_custom/fla_npu/fla_npu/ops/ascendc/_aclnn_ctypes.py:1534-1783) and defers the rest to a third-party
// package; the gradients here are those of the recurrence itself
// (tests/atk/recurrent_kda/executor_recurrent_kda.py:63-83), derived for the anchored chunk form of the forward:
//   gk = chunk cumsum(g), a = gk at the middle token, Qp = Q e^{gk-a}, Kp = K e^{gk-a}, Kn = K e^{a-gk},
//   P = tril(Qp Kn^T), M = strict_tril(Kp Kn^T), X = (I + beta M)^-1, Sa = diag(e^a) S, D = e^{gk_L-a}:
//   Vn = X (beta (V - Kp Sa)),  O = scale (Qp Sa + P Vn),  S' = diag(D) (Sa + Kn^T Vn).
// The entry point recomputes the forward (prep -> inverse -> forward scan, saving Sa and Vn as strip images) and runs
//
//  kda_scan_bwd_kernel  (kda_scan_bwd.cuh; reverse-sequential over chunks, one CTA per (sequence, value head, 128 channels of V)):
//      dS'a = diag(D) dS'          dVn = scale P^T dO + Kn dS'a          dZ = X^T dVn          dV = beta dZ
//      dSa  = dS'a + Qp^T (scale dO) + Kp^T (-beta dZ)                   dS = diag(e^a) dSa    dh0 = dS after the first chunk
//  kda_bwd_par_kernel  (parallel over chunks, one CTA per (chunk, q/k head), looping over the value heads of the group):
//      dP = scale tril(dO Vn^T)     dA = -strict_tril(dZ Vn^T)     dM = beta dA
//      dQp = scale dO Sa^T + dP Kn          dKp = -beta dZ Sa^T + dM Kn          dKn = Vn dS'a^T + dP^T Qp + dM^T Kp
//      dq = dQp e^{gk-a}     dk = dKp e^{gk-a} + dKn e^{a-gk}     dbeta = sum_v dZ V - Kp.(dZ Sa^T) + sum_j dA M
//      dgk = Qp dQp + Kp dKp - Kn dKn;  dgk_L += sum_v dS'a Sa + sum_i Kn_i (Vn dS'a^T)_i;  dg = reverse chunk cumsum(dgk)
//
// Every operand that is not an exact bf16 input travels as bf16 hi + bf16 residual (three tcgen05.mma passes);
// accumulation is fp32 in TMEM.
#include <algorithm>
#include "gdn_common.cuh"
#include "fla_b200_internal.h"
#include "kernel_timer.h"
#include "aux_stream.h"
#include "kda_common.cuh"
#include "scan_segments.cuh"
#include "tensor_map.h"

namespace fla {

struct KdaBwdParams {
  const bf16* v; const bf16* dO; const void* beta;
  const bf16* q; const bf16* k;               // raw rows, read only when dq / dk go through the normalisation:
  const float* q_rstd; const float* k_rstd;   // [tokens, HK] or null
  int64_t q_st, q_sh, k_st, k_sh;
  const bf16* qk_img; const bf16* kn_img; const bf16* p_img; const bf16* x_img;
  const float* vec; const float* gk;
  const bf16* s_img; const bf16* vn_img;
  bf16* ds_img;        // [chunks, HV, V/64, {hi, lo}, 16 strips of 8 key dims, 64 channels]  dS'a entering each chunk
  bf16* dz_img;        // [chunks, HV, V/64, {dO, dZ hi, dZ lo}, 8 strips of 8 tokens, 64 channels]
  const bf16* seg_m;   // split chains: the forward's transition matrices
  float* seg_dh;       // split chains: [segments, HV, V/128, 128, 128]
  int seg_len;         // chunks per segment
  int* counter;        // tiles the par kernel has handed out beyond its first wave; the scan in front of it sets it to zero
  int clear;           // the scan is the call's first kernel: it clears the status word
  float* bz;           // [V/32, tokens, HV] partial sums of dZ * V over the 32-column slices of V
  const float* dht; float* dh0;
  void* dq; void* dk; void* dv; void* dg; void* dbeta;
  const int32_t* cu_seqlens; const int32_t* chunk_offsets;
  int64_t v_st, v_sh, do_st, do_sh, beta_st;
  int64_t dq_st, dq_sh, dk_st, dk_sh, dv_st, dv_sh, dg_st, dg_sh;
  int64_t total_tokens;
  int N, T, HK, HV, beta_is_f32;
  int dq_f32, dk_f32, dv_f32, dg_f32, dbeta_f32;   // gradients leave in the dtypes of their inputs: f32, else bf16
  int n0, n1;          // sequences of this launch (the backward may be launched as two halves of the batch)
  int V, nvb;          // value head dim (128 or 256) and its number of 64-column blocks
  float scale;
  int* status;
};

constexpr int64_t kKdaDsImg = 16384, kKdaDzImg = 12288;   // bf16 elements per (chunk, head, 64-column block of V)

}  // namespace fla
#include "kda_scan_bwd.cuh"
namespace fla {

// ============================================================================================= par
constexpr uint32_t qOffQKH = 0, qOffQKL = 32768, qOffKNH = 65536, qOffKNL = 81920;       // per-head operand images
// Operands of one 64-channel step are strips (sm100.cuh) whose 64 rows are value channels, the reduction dim of its products.
constexpr uint32_t qOffAL = 98304;              // 8 KB of zeros (dO has no residual), then dZ_lo^T
constexpr uint32_t qOffAH = 114688;             // [dO^T | dZ_hi^T]: 16 strips of 8 tokens
constexpr uint32_t qOffVNH = 131072, qOffVNL = 139264;
constexpr uint32_t qOffSH = 147456, qOffSL = 163840, qOffDSH = 180224, qOffDSL = 196608;
constexpr uint32_t kKdaParSmem = 212992;
// What reuses the step buffers (all but the zeros): the [dP; dM] panels and the chunk's gk rows (four 64 x 32 fp32 TMA tiles,
// swizzled), then, over the panels, two fp32 [64][132] tiles of the dg assembly.
constexpr uint32_t qOffPAH = qOffAL + 8192, qOffPAL = qOffPAH + 16384;
constexpr uint32_t qOffTile = qOffPAH;
constexpr int kTileStride = 132;   // 16-byte aligned rows; float4 row stores and float2 column reads are both conflict-free
constexpr uint32_t kTileBytes = kC * kTileStride * 4;
constexpr uint32_t qOffGk = qOffTile + 2 * kTileBytes;
static_assert(qOffGk % 1024 == 0 && qOffGk + 32768 <= kKdaParSmem && qOffGk >= qOffPAL + 16384, "dg tiles, panels and gk rows must fit in the step buffers");
constexpr uint32_t qColQK = 0, qColDV = 64, qColTA = 128, qColTB1 = 256, qColTB2 = 384;
constexpr uint32_t qColTA2 = 0;                 // [dP; dM] Kn, where the two score tiles were
constexpr uint32_t kKdaStepBytes = 16384 + 8192 + 16384 + 32768 + 32768;
constexpr int kParWorkers = 512, kParThreads = kParWorkers + 32;

// sum over 8 columns of (hi + lo panel values) * x
__device__ __forceinline__ void chunk_vals(const uint8_t* pan_hi, const uint8_t* pan_lo, int row, int ch, float* f) {
  float lo[8];
  unpack_bf16x8(*reinterpret_cast<const uint4*>(pan_hi + panel_chunk_off(row, ch)), f);
  unpack_bf16x8(*reinterpret_cast<const uint4*>(pan_lo + panel_chunk_off(row, ch)), lo);
#pragma unroll
  for (int j = 0; j < 8; ++j) f[j] += lo[j];
}

// Sum over the 32 lanes of each of 8 per-lane values: lanes 4 j .. 4 j + 3 end up with the total of value j.
// Recursive halving: at every step a lane keeps one half of its values and hands the other half to its partner.
__device__ __forceinline__ float warp_column_sums8(const float (&v)[8], int lane) {
  float a[4], b[2];
#pragma unroll
  for (int i = 0; i < 4; ++i) a[i] = ((lane & 16) ? v[4 + i] : v[i]) + __shfl_xor_sync(0xffffffffu, (lane & 16) ? v[i] : v[4 + i], 16);
#pragma unroll
  for (int i = 0; i < 2; ++i) b[i] = ((lane & 8) ? a[2 + i] : a[i]) + __shfl_xor_sync(0xffffffffu, (lane & 8) ? a[i] : a[2 + i], 8);
  float r = ((lane & 4) ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, (lane & 4) ? b[0] : b[1], 4);
  r += __shfl_xor_sync(0xffffffffu, r, 2);
  return r + __shfl_xor_sync(0xffffffffu, r, 1);
}

__device__ __forceinline__ void par_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kParWorkers) : "memory"); }
__device__ __forceinline__ bool par_sync_and(bool ok) {
  uint32_t r;
  asm volatile(
      "{\n"
      " .reg .pred p, q;\n"
      " setp.ne.u32 q, %1, 0;\n"
      " bar.red.and.pred p, 1, %2, q;\n"
      " selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(r)
      : "r"(uint32_t(ok)), "n"(kParWorkers)
      : "memory");
  return r != 0;
}

// One CTA per SM; sixteen worker warps and one thread that issues every load and product.  An item is one value head of one
// (chunk, q/k head) tile; the workers' phases of an item and what the issuing thread does meanwhile:
//     sum dS'a Sa            score product, then per 64 channels of V: load, three products
//     [dP; dM] operand       -
//     -                      the products with [dP; dM], gk rows
//     dq, dk, dg tiles       -                                            (images free: the next item's are requested)
//     dg, dq, dk out         score product of the next item, its first step's loads
// What bounded the one-tile-per-CTA form with eight warps (40,000 cycles a tile, of which the tensor core needs 10,000 and HBM 17,000): nothing
// overlapped - the prologue and the first loads (5,400), two V steps (9,000), the products with [dP; dM] behind the issuing thread's own
// epilogue work (5,000), eight warps' worth of fp32 epilogues (12,000), stores (3,000).
// 32,768 tokens of 32 heads: 2.36 -> 1.78 ms.
// Tiles are handed out by a counter: next to the other half of the batch's scan (below) the CTAs do not start together.
// NVB: 64-column blocks of V per head (2 or 4), a compile-time trip count that keeps the block loop unrolled.  NORM: dq, dk go through
// the q/k normalisation at the end (a kernel of its own: the epilogue's registers would spill in the other).
template <int NVB, bool NORM>
__global__ void __launch_bounds__(kParThreads, 1) kda_bwd_par_kernel(KdaBwdParams p, int chunks, const __grid_constant__ CUtensorMap tm_gk) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(16) float anchor_s[kK], beta_s[kK];      // neighbours in the prep kernel's record: one load
  __shared__ float red[2][4][kC];      // rkG, ma : [32-column group of the row][row]
  __shared__ float sds_s[kK];          // sum_v dS'a * Sa per key channel
  __shared__ __align__(8) float colsum_s[8][kK];    // per 8-row part: column sums of the dgk tiles
  __shared__ float ndot_s[NORM ? 4 : 1][2 * kC];    // q.dq / k.dk of the complete rows, per 32-column group (normalised q, k only)
  __shared__ float t1col_s[2][kK];     // per 32-row quadrant: sum_i Kn_i (Vn dS'a^T)_i of the last-row term
  __shared__ int item_s, tok0_s;
  __shared__ uint32_t tmem_base_s;
  __shared__ __align__(8) uint64_t img_bar, load_bar, gk_bar;            // loads
  __shared__ __align__(8) uint64_t step_bar, p1_bar, mma2_bar;           // products: a V step, the last V step, those with [dP; dM]
  __shared__ __align__(8) uint64_t sds_bar, epi1_bar, epi2_bar, dg_bar;  // workers: step buffers read, [dP; dM] there, images and accumulators read, tiles read

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
    for (uint64_t* b : {&img_bar, &load_bar, &gk_bar, &step_bar, &p1_bar, &mma2_bar}) mbar_init(b, 1);
    for (uint64_t* b : {&sds_bar, &epi1_bar, &epi2_bar, &dg_bar}) mbar_init(b, kParWorkers / 32);
    mbar_init_fence();
    tma_prefetch_descriptor(&tm_gk);
  }
  if (tid < kParWorkers) *reinterpret_cast<uint4*>(smem + qOffAL + tid * 16) = make_uint4(0, 0, 0, 0);
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = tmem_base_s;
  const uint32_t sb = smem_u32(smem);

  if (warp == kParWorkers / 32) {
    if (lane == 0) {
      auto record = [&](int tile, int h) { return int64_t(flat0 + tile / p.HK) * p.HV + (tile % p.HK) * G + h; };
      auto issue_images = [&](int64_t cidx) {           // [Qp; Kp], Kn, the anchor and beta of one value head
        mbar_arrive_expect_tx(&img_bar, 65536 + 32768 + 1024);
        bulk_load(sb + qOffQKH, p.qk_img + cidx * kKdaQkImg, 65536, &img_bar);
        bulk_load(sb + qOffKNH, p.kn_img + cidx * kKdaKnImg, 32768, &img_bar);
        bulk_load(smem_u32(anchor_s), p.vec + cidx * kKdaVecs * kK + 2 * kK, 512, &img_bar);
        bulk_load(smem_u32(beta_s), p.vec + cidx * kKdaVecs * kK + 3 * kK, 512, &img_bar);
      };
      auto issue_loads = [&](int64_t cidx, int vb) {    // operands of one (value head, V block) step
        mbar_arrive_expect_tx(&load_bar, kKdaStepBytes);
        const bf16* dz = p.dz_img + (cidx * NVB + vb) * kKdaDzImg;
        bulk_load(sb + qOffAH, dz, 16384, &load_bar);
        bulk_load(sb + qOffAL + 8192, dz + 8192, 8192, &load_bar);
        bulk_load(sb + qOffVNH, p.vn_img + (cidx * NVB + vb) * kKdaVnImg, 16384, &load_bar);
        bulk_load(sb + qOffSH, p.s_img + (cidx * NVB + vb) * kKdaSImg, 32768, &load_bar);
        bulk_load(sb + qOffDSH, p.ds_img + (cidx * NVB + vb) * kKdaDsImg, 32768, &load_bar);
      };
      const Operand opQKh{sb + qOffQKH, 16384, 0}, opQKl{sb + qOffQKL, 16384, 0};           // [Qp; Kp], reduction over key dims
      const Operand opQKnh{sb + qOffQKH, 16384, 1}, opQKnl{sb + qOffQKL, 16384, 1};         // as B, N = 128 key dims, reduction over 128 rows
      const Operand opKNbh{sb + qOffKNH, 8192, 0}, opKNbl{sb + qOffKNL, 8192, 0};           // Kn as B, N = 64 tokens
      const Operand opKNnh{sb + qOffKNH, 8192, 1}, opKNnl{sb + qOffKNL, 8192, 1};           // Kn as B, N = 128 key dims, reduction over tokens
      const Operand opAH{sb + qOffAH, 1024, 2}, opAL{sb + qOffAL, 1024, 2};                 // [dO; dZ], M = 128 tokens
      const Operand opVNbH{sb + qOffVNH, 1024, 2}, opVNbL{sb + qOffVNL, 1024, 2};           // Vn as B (N = 64 tokens)
      const Operand opVNaH{sb + qOffVNH - 8192, 1024, 2}, opVNaL{sb + qOffVNL - 8192, 1024, 2};  // Vn as A, valid rows 64..127
      const Operand opSH{sb + qOffSH, 1024, 2}, opSL{sb + qOffSL, 1024, 2};                 // Sa block as B (N = 128 key dims)
      const Operand opDSH{sb + qOffDSH, 1024, 2}, opDSL{sb + qOffDSL, 1024, 2};
      const Operand opPAH{sb + qOffPAH, 16384, 0}, opPAL{sb + qOffPAL, 16384, 0};           // [dP; dM], reduction over j
      const Operand opPATh{sb + qOffPAH - 8192, 8192, 1}, opPATl{sb + qOffPAL - 8192, 8192, 1};  // its transpose, valid rows 64..127

      auto wait = [&](uint64_t* bar, uint32_t& phase) {
        const bool r = mbar_wait(bar, phase, p.status, FLA_ERR_TIMEOUT);
        phase ^= 1;
        return r;
      };
      uint32_t ph_img = 0, ph_load = 0, ph_step = 0, ph_p1 = 0, ph_sds = 0, ph_epi1 = 0, ph_epi2 = 0, ph_dg = 0;
      int tile = blockIdx.x, h = 0;
      bool ok = true;
      if (tile < tiles) {
        const int64_t cidx = record(tile, 0);
        item_s = tile * G;
        issue_images(cidx);
        issue_loads(cidx, 0);
      } else {
        item_s = -1;
        mbar_arrive_expect_tx(&img_bar, 0);
        ok = false;
      }
      int after = ok ? int(gridDim.x) + atomicAdd(p.counter, 1) : 0;      // the tile that follows
      while (ok) {
        const int64_t cidx = record(tile, h);
        const int hv = (tile % p.HK) * G + h;
        if (!wait(&img_bar, ph_img)) break;
        tc_fence_after();
        mma_tile(tbase + qColQK, opQKh, opKNbh, 128, 64, 8, false);
        mma_tile(tbase + qColQK, opQKh, opKNbl, 128, 64, 8, true);
        mma_tile(tbase + qColQK, opQKl, opKNbh, 128, 64, 8, true);
        for (int vb = 0; vb < NVB && ok; ++vb) {
          ok = wait(&load_bar, ph_load);
          if (!ok) break;
          const bool accf = vb > 0;
          // [dO; dZ] . [Vn_lo | Sa_hi]^T as one N = 192 product: the two images are neighbours in shared memory and their
          // accumulators neighbours in tensor memory, so the A operand is read once for both
          static_assert(qOffVNL + 8192 == qOffSH && qColDV + 64 == qColTA, "the N = 192 product needs both pairs adjacent");
          mma_tile(tbase + qColDV, opAH, opVNbL, 128, 192, 4, accf);
          mma_tile(tbase + qColDV, opAH, opVNbH, 128, 64, 4, true);
          mma_tile(tbase + qColDV, opAL, opVNbH, 128, 64, 4, true);
          mma_tile(tbase + qColTA, opAH, opSL, 128, 128, 4, true);
          mma_tile(tbase + qColTA, opAL, opSH, 128, 128, 4, true);
          mma_tile(tbase + qColTB1, opVNaH, opDSH, 128, 128, 4, accf);
          mma_tile(tbase + qColTB1, opVNaH, opDSL, 128, 128, 4, true);
          mma_tile(tbase + qColTB1, opVNaL, opDSH, 128, 128, 4, true);
          if (vb + 1 < NVB) {
            mma_commit(&step_bar);
            ok = wait(&sds_bar, ph_sds) && wait(&step_bar, ph_step);
            if (ok) issue_loads(cidx, vb + 1);
          } else {
            mma_commit(&p1_bar);
            ok = wait(&sds_bar, ph_sds) && wait(&p1_bar, ph_p1);
            if (ok) {   // the step buffers are free: this head's gk rows, channels 32 b .. 32 b + 31 in tile b
              mbar_arrive_expect_tx(&gk_bar, 4 * 8192);
#pragma unroll
              for (int b = 0; b < 4; ++b) tma_load_tile(sb + qOffGk + b * 8192, &tm_gk, 32 * b, hv, tok0_s, &gk_bar);
            }
          }
        }
        if (!ok || !wait(&epi1_bar, ph_epi1)) break;
        // TA2 = [dP; dM] Kn   and   TB2 = [dP^T | dM^T] [Qp; Kp]
        tc_fence_after();
        mma_tile(tbase + qColTA2, opPAH, opKNnh, 128, 128, 4, false);
        mma_tile(tbase + qColTA2, opPAH, opKNnl, 128, 128, 4, true);
        mma_tile(tbase + qColTA2, opPAL, opKNnh, 128, 128, 4, true);
        mma_tile(tbase + qColTB2, opPATh, opQKnh, 128, 128, 8, false);
        mma_tile(tbase + qColTB2, opPATh, opQKnl, 128, 128, 8, true);
        mma_tile(tbase + qColTB2, opPATl, opQKnh, 128, 128, 8, true);
        mma_commit(&mma2_bar);
        if (++h == G) {
          h = 0;
          tile = after;
          if (tile < tiles) after = int(gridDim.x) + atomicAdd(p.counter, 1);
        }
        const bool more = tile < tiles;
        if (!wait(&epi2_bar, ph_epi2)) break;
        item_s = more ? tile * G + h : -1;
        if (!more) {
          mbar_arrive_expect_tx(&img_bar, 0);
          break;
        }
        issue_images(record(tile, h));
        if (!wait(&dg_bar, ph_dg)) break;
        issue_loads(record(tile, h), 0);
      }
    }
  } else {
    const int quad = warp & 3, cg = warp >> 2;  // my 32 accumulator rows, my 32 key-dim columns
    const int row = quad * 32 + lane;           // accumulator row == TMEM lane
    const bool kside = quad >= 2;
    const int tok = row & 63;
    const uint32_t trow = tmem_addr(tbase, quad * 32, 0);
    float* tile_q = reinterpret_cast<float*>(smem + qOffTile);
    float* tile_k = reinterpret_cast<float*>(smem + qOffTile + kTileBytes);
    const uint8_t* qk_h = smem + qOffQKH + (cg >> 1) * 16384;      // the panels of my columns
    const uint8_t* qk_l = smem + qOffQKL + (cg >> 1) * 16384;
    const uint8_t* kn_h = smem + qOffKNH + (cg >> 1) * 8192;
    const uint8_t* kn_l = smem + qOffKNL + (cg >> 1) * 8192;
    auto signal = [&](uint64_t* bar) {      // my warp is done with what the barrier stands for
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    uint32_t ph_load = 0, ph = 0;
    bool ok = true;
    float acc[32];      // running dq (q-side rows) or dk (k-side rows), my 32 key-dim columns
#pragma unroll
    for (int i = 0; i < 32; ++i) acc[i] = 0.f;

    while (true) {
      // a wait that runs out makes this thread skip the rest of its waits; all leave together at the next turn
      ok = ok && mbar_wait(&img_bar, ph, p.status, FLA_ERR_TIMEOUT);
      const int item = item_s;
      if (!par_sync_and(ok) || item < 0) break;
      const int tile = item / G, h = item - tile * G, hk = tile % p.HK, hv = hk * G + h;
      const ChunkPos pos = chunk_pos(p.cu_seqlens, p.chunk_offsets, p.N, p.T, p.n0, chunk0 + tile / p.HK);
      const int t0 = pos.c * kC, rows = min(kC, pos.sq.len - t0);
      const int64_t tok0 = int64_t(pos.sq.bos) + t0;
      if (tid == 0) tok0_s = int(tok0);
      float bz = 0.f;
      if (tid < rows) {
        const int64_t gidx = (tok0 + tid) * p.HV + hv, bzs = p.total_tokens * p.HV;
#pragma unroll
        for (int s = 0; s < 2 * NVB; ++s) bz += p.bz[s * bzs + gidx];
      }
      {      // sum_v dS'a * Sa per key channel while the products run: strip `warp` is 8 key dims
        float sds[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) sds[j] = 0.f;
        for (int vb = 0; vb < NVB; ++vb) {
          ok = ok && mbar_wait(&load_bar, ph_load, p.status, FLA_ERR_TIMEOUT);
          ph_load ^= 1;
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const uint32_t off = warp * 1024 + (lane + r * 32) * 16;
            float s1[8], s2[8], d1[8], d2[8];
            unpack_bf16x8(*reinterpret_cast<const uint4*>(smem + qOffSH + off), s1);
            unpack_bf16x8(*reinterpret_cast<const uint4*>(smem + qOffSL + off), s2);
            unpack_bf16x8(*reinterpret_cast<const uint4*>(smem + qOffDSH + off), d1);
            unpack_bf16x8(*reinterpret_cast<const uint4*>(smem + qOffDSL + off), d2);
#pragma unroll
            for (int j = 0; j < 8; ++j) sds[j] += (s1[j] + s2[j]) * (d1[j] + d2[j]);
          }
          signal(&sds_bar);
        }
        const float t = warp_column_sums8(sds, lane);
        if (!(lane & 3)) sds_s[warp * 8 + (lane >> 2)] = t;
      }

      // ---- epilogue 1: score-tile gradients -> [dP; dM] operand
      ok = ok && mbar_wait(&p1_bar, ph, p.status, FLA_ERR_TIMEOUT);
      tc_fence_after();
      const float beta_i = beta_s[tok];
      float rkG = 0.f;
      {
        float sc[16], dvv[16], ma = 0.f;
        tmem_ld16(trow + qColQK + cg * 16, sc);
        tmem_ld16(trow + qColDV + cg * 16, dvv);
        tmem_ld_wait();
        if (!kside) {
#pragma unroll
          for (int jj = 0; jj < 16; ++jj) dvv[jj] = (cg * 16 + jj <= tok) ? p.scale * dvv[jj] : 0.f;
        } else {
#pragma unroll
          for (int jj = 0; jj < 16; ++jj) {
            const bool keep = cg * 16 + jj < tok;
            const float dA = keep ? -dvv[jj] : 0.f;
            ma += keep ? dA * sc[jj] : 0.f;      // select: entries above the diagonal of M may be huge
            dvv[jj] = dA * beta_i;
          }
          red[1][cg][tok] = ma;
        }
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {
          uint4 hi, lo;
          split8(dvv + ch * 8, hi, lo);
          const uint32_t off = panel_chunk_off(row, cg * 2 + ch);
          *reinterpret_cast<uint4*>(smem + qOffPAH + off) = hi;
          *reinterpret_cast<uint4*>(smem + qOffPAL + off) = lo;
        }
      }
      fence_async_smem();
      tc_fence_before();
      signal(&epi1_bar);

      // ---- epilogue 2: dq / dk rows of this head and the two dg tiles (the panels are free then)
      ok = ok && mbar_wait(&gk_bar, ph, p.status, FLA_ERR_TIMEOUT) && mbar_wait(&mma2_bar, ph, p.status, FLA_ERR_TIMEOUT);
      tc_fence_after();
      const bool live = tok < rows;
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) {
        const int c8 = cg * 32 + ch * 8, pc = (cg & 1) * 4 + ch;      // my 8 columns, their 16-byte piece of the panel row
        float x[8], x2[8], gv[8];
        tmem_ld8(trow + qColTA + c8, x);
        tmem_ld8(trow + qColTA2 + c8, x2);
        {
          const uint8_t* gt = smem + qOffGk + cg * 8192 + tok * 128;
          const float4 g0 = *reinterpret_cast<const float4*>(gt + (((2 * ch) ^ (tok & 7)) << 4));
          const float4 g1 = *reinterpret_cast<const float4*>(gt + (((2 * ch + 1) ^ (tok & 7)) << 4));
          float an[8];
          gather8(anchor_s + c8, an);
          gv[0] = g0.x; gv[1] = g0.y; gv[2] = g0.z; gv[3] = g0.w; gv[4] = g1.x; gv[5] = g1.y; gv[6] = g1.z; gv[7] = g1.w;
#pragma unroll
          for (int j = 0; j < 8; ++j) gv[j] = (gv[j] - an[j]) * kLog2e;
        }
        float tv[8];
        if (!kside) {
          float qp[8];
          chunk_vals(qk_h, qk_l, tok, pc, qp);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float xv = p.scale * x[j] + x2[j];
            acc[ch * 8 + j] += live ? xv * exp2_fast(gv[j]) : 0.f;
            tv[j] = live ? qp[j] * xv : 0.f;
          }
        } else {
          float y1[8], y2[8], kp[8], kn[8], t1v[8];
          tmem_ld8(trow + qColTB1 + c8, y1);
          tmem_ld8(trow + qColTB2 + c8, y2);
          chunk_vals(qk_h, qk_l, 64 + tok, pc, kp);
          chunk_vals(kn_h, kn_l, tok, pc, kn);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            rkG += kp[j] * x[j];      // Kp_i . (dZ Sa^T)_i
            const float dkp = x2[j] - beta_i * x[j], dkn = y1[j] + y2[j];
            acc[ch * 8 + j] += live ? dkp * exp2_fast(gv[j]) + dkn * exp2_fast(-gv[j]) : 0.f;
            tv[j] = live ? kp[j] * dkp - kn[j] * dkn : 0.f;
            t1v[j] = live ? kn[j] * y1[j] : 0.f;
          }
          // last-row term: column sums of Kn * (Vn dS'a^T) over my warp's 32 rows
          const float t = warp_column_sums8(t1v, lane);
          if (!(lane & 3)) t1col_s[quad - 2][c8 + (lane >> 2)] = t;
        }
        float* dst = (kside ? tile_k : tile_q) + tok * kTileStride + c8;
        *reinterpret_cast<float4*>(dst) = make_float4(tv[0], tv[1], tv[2], tv[3]);
        *reinterpret_cast<float4*>(dst + 4) = make_float4(tv[4], tv[5], tv[6], tv[7]);
      }
      if (kside) red[0][cg][tok] = rkG;
      tc_fence_before();
      signal(&epi2_bar);
      ok = par_sync_and(ok);
      // dg = reverse chunk-local cumulative sum of dgk; the last row additionally carries
      // sum_v dS'a Sa + sum_i Kn_i (Vn dS'a^T)_i, which therefore reaches every row.
      {
        // A thread has two key channels and 8 rows: local totals first, then the suffix sums.
        const int kc = (tid & 63) * 2, part = tid >> 6, r0 = part * 8;
        float2 v[8];      // rows past the end hold zeros
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float2 a = *reinterpret_cast<const float2*>(tile_q + (r0 + i) * kTileStride + kc);
          const float2 b = *reinterpret_cast<const float2*>(tile_k + (r0 + i) * kTileStride + kc);
          v[i] = make_float2(a.x + b.x, a.y + b.y);
        }
        float2 run = make_float2(sds_s[kc] + t1col_s[0][kc] + t1col_s[1][kc], sds_s[kc + 1] + t1col_s[0][kc + 1] + t1col_s[1][kc + 1]);
        float db = 0.f;
        if (tid < kC) {
          db = bz;
#pragma unroll
          for (int s = 0; s < 4; ++s) db += red[1][s][tid] - red[0][s][tid];
        }
        fence_async_smem();
        signal(&dg_bar);
#pragma unroll
        for (int i = 6; i >= 0; --i) {      // suffix sums of my rows
          v[i].x += v[i + 1].x;
          v[i].y += v[i + 1].y;
        }
        *reinterpret_cast<float2*>(&colsum_s[part][kc]) = v[0];
        if (tid < rows) {
          const int64_t gidx = (tok0 + tid) * p.HV + hv;
          if (p.dbeta_f32) static_cast<float*>(p.dbeta)[gidx] = db;
          else static_cast<bf16*>(p.dbeta)[gidx] = __float2bfloat16_rn(db);
        }
        par_sync();
        for (int s = part + 1; s < 8; ++s) {
          const float2 t = *reinterpret_cast<const float2*>(&colsum_s[s][kc]);
          run.x += t.x;
          run.y += t.y;
        }
        const int64_t base = tok0 * p.dg_st + hv * p.dg_sh + kc;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int t = r0 + i;
          if (ok && t < rows) {
            if (p.dg_f32) *reinterpret_cast<float2*>(static_cast<float*>(p.dg) + base + t * p.dg_st) = make_float2(run.x + v[i].x, run.y + v[i].y);
            else *reinterpret_cast<uint32_t*>(static_cast<bf16*>(p.dg) + base + t * p.dg_st) = pack_bf16(run.x + v[i].x, run.y + v[i].y);
          }
        }
      }
      ph ^= 1;
      if (h + 1 < G) continue;

      if constexpr (NORM) {   // the rows are complete: rstd (dx - x (x . dx)) with x the normalised row, made again from the raw one
        const int64_t r = tok0 + min(tok, rows - 1);
        const float rs = (kside ? p.k_rstd : p.q_rstd)[r * p.HK + hk];
        const bf16* src = (kside ? p.k + r * p.k_st + hk * p.k_sh : p.q + r * p.q_st + hk * p.q_sh) + cg * 32;
        uint4 raw[4];
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) raw[ch] = *reinterpret_cast<const uint4*>(src + ch * 8);
        float t = 0.f;
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
          float f[8];
          unpack_bf16x8(raw[ch], f);
#pragma unroll
          for (int j = 0; j < 8; ++j) f[j] = f[j] * rs;
          raw[ch] = pack8(f);
          unpack_bf16x8(raw[ch], f);
#pragma unroll
          for (int j = 0; j < 8; ++j) t += f[j] * acc[ch * 8 + j];
        }
        ndot_s[cg][row] = t;
        par_sync();
        t = (ndot_s[0][row] + ndot_s[1][row]) + (ndot_s[2][row] + ndot_s[3][row]);
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
          float f[8];
          unpack_bf16x8(raw[ch], f);
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[ch * 8 + j] = (acc[ch * 8 + j] - t * f[j]) * rs;
        }
      }
      if (ok && live) {
        void* base = kside ? p.dk : p.dq;
        const int64_t off = (kside ? (tok0 + tok) * p.dk_st + hk * p.dk_sh : (tok0 + tok) * p.dq_st + hk * p.dq_sh) + cg * 32;
        if (kside ? p.dk_f32 : p.dq_f32) {
          float* dst = static_cast<float*>(base) + off;
#pragma unroll
          for (int i = 0; i < 32; i += 4) *reinterpret_cast<float4*>(dst + i) = make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
        } else {
          bf16* dst = static_cast<bf16*>(base) + off;
#pragma unroll
          for (int ch = 0; ch < 4; ++ch) *reinterpret_cast<uint4*>(dst + ch * 8) = pack8(acc + ch * 8);
        }
      }
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

// Workspace: status | [forward workspace | gk | s_img | vn_img unless the caller passes the forward's saved buffer] | ds_img | dz_img | bz
static uint64_t kda_bwd_ws_layout(int64_t total_chunks, int64_t HV, int64_t nvb, int64_t tokens, bool have_saved, const SegPlan& plan,
                                  uint64_t* off_saved, uint64_t off[4]) {
  const uint64_t per = uint64_t(total_chunks) * HV;
  uint64_t o = 256, so[5];
  *off_saved = o;
  if (!have_saved) o += align_up(kda_saved_layout(total_chunks, HV, nvb, tokens, plan.split ? plan.count : 0, so), 256);
  off[0] = o; o += align_up(per * nvb * kKdaDsImg * 2, 256);
  off[1] = o; o += align_up(per * nvb * kKdaDzImg * 2, 256);
  off[2] = o; o += align_up(uint64_t(2 * nvb) * tokens * HV * 4, 256);
  off[3] = o;      // H of the recomputed forward, then dH
  if (plan.split) o += uint64_t(plan.count) * HV * (nvb / 2) * kSegHBytes;
  return o;
}

static int kda_bwd_geometry(const fla_kda_chunk_bwd_args* a, int64_t* total_chunks, int* N) {
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

static SegPlan kda_bwd_plan(const fla_kda_chunk_bwd_args* a, int64_t total_chunks, int N) {      // that of the forward
  const bool packed = a->cu_seqlens.data != nullptr;
  return scan_plan(N, total_chunks, packed ? a->max_seqlen : a->q.shape[1], packed, a->v.shape[2], a->v.shape[3]);
}

extern "C" FLA_API int fla_b200_kda_chunk_bwd_workspace_size(const fla_kda_chunk_bwd_args* a, uint64_t* bytes) {
  if (!a || !bytes) return FLA_ERR_NULL;
  int64_t total_chunks; int N;
  const int st = kda_bwd_geometry(a, &total_chunks, &N);
  if (st) return st;
  uint64_t off[4], off_saved;
  const int64_t V = a->v.shape[3];
  if (V != kV && V != 2 * kV) return FLA_ERR_SHAPE;
  *bytes = kda_bwd_ws_layout(total_chunks, a->v.shape[2], V / kBV, a->q.shape[0] * a->q.shape[1], a->saved.data != nullptr,
                             kda_bwd_plan(a, total_chunks, N), &off_saved, off);
  return FLA_OK;
}

static int kda_bwd_check_tok(const fla_tensor_t& t, int64_t B, int64_t T, int64_t heads, int64_t dim, bool allow_f32) {
  if (!t.data) return FLA_ERR_NULL;
  if (t.ndim != 4 || t.shape[0] != B || t.shape[1] != T || t.shape[2] != heads || t.shape[3] != dim) return FLA_ERR_SHAPE;
  if (t.dtype != FLA_BF16 && !(allow_f32 && t.dtype == FLA_F32)) return FLA_ERR_DTYPE;
  const int64_t esz = t.dtype == FLA_F32 ? 4 : 2;
  if (t.stride[3] != 1 || (t.stride[2] * esz) % 16 || (t.stride[1] * esz) % 16 || !aligned16(t.data)) return FLA_ERR_LAYOUT;
  if (B > 1 && t.stride[0] != T * t.stride[1]) return FLA_ERR_LAYOUT;
  return FLA_OK;
}
static int kda_bwd_check_tok3(const fla_tensor_t& t, int64_t B, int64_t T, int64_t heads, bool dense) {
  if (!t.data) return FLA_ERR_NULL;
  if (t.ndim != 3 || t.shape[0] != B || t.shape[1] != T || t.shape[2] != heads) return FLA_ERR_SHAPE;
  if (t.dtype != FLA_BF16 && t.dtype != FLA_F32) return FLA_ERR_DTYPE;
  if (t.stride[2] != 1 || (B > 1 && t.stride[0] != T * t.stride[1])) return FLA_ERR_LAYOUT;
  if (dense && t.stride[1] != heads) return FLA_ERR_LAYOUT;
  return FLA_OK;
}

extern "C" FLA_API int fla_b200_kda_chunk_bwd(const fla_kda_chunk_bwd_args* a, void* workspace, uint64_t workspace_bytes,
                                              void* stream) {
  if (!a) return FLA_ERR_NULL;
  int64_t total_chunks; int N;
  int st = kda_bwd_geometry(a, &total_chunks, &N);
  if (st) return st;
  const int64_t B = a->q.shape[0], T = a->q.shape[1], HK = a->q.shape[2], HV = a->v.shape[2];
  if (HK <= 0 || HV <= 0 || HV % HK) return FLA_ERR_SHAPE;
  const int64_t V = a->v.shape[3], nvb = V / kBV;
  if (V != kV && V != 2 * kV) return FLA_ERR_SHAPE;
  if ((st = kda_bwd_check_tok(a->q, B, T, HK, kK, false))) return st;
  if ((st = kda_bwd_check_tok(a->k, B, T, HK, kK, false))) return st;
  if ((st = kda_bwd_check_tok(a->v, B, T, HV, V, false))) return st;
  if ((st = kda_bwd_check_tok(a->g, B, T, HV, kK, true))) return st;
  if ((st = kda_bwd_check_tok(a->d_o, B, T, HV, V, false))) return st;
  if ((st = kda_bwd_check_tok(a->dq, B, T, HK, kK, true))) return st;
  if ((st = kda_bwd_check_tok(a->dk, B, T, HK, kK, true))) return st;
  if ((st = kda_bwd_check_tok(a->dv, B, T, HV, V, true))) return st;
  if ((st = kda_bwd_check_tok(a->dg, B, T, HV, kK, true))) return st;
  if ((st = kda_bwd_check_tok3(a->beta, B, T, HV, false))) return st;
  if ((st = kda_bwd_check_tok3(a->dbeta, B, T, HV, true))) return st;
  for (const fla_tensor_t* s : {&a->initial_state, &a->dht, &a->dh0}) {
    if (!s->data) continue;
    if (s->dtype != FLA_F32) return FLA_ERR_DTYPE;
    if (s->ndim != 4 || s->shape[0] != N || s->shape[1] != HV || s->shape[2] != kK || s->shape[3] != V) return FLA_ERR_SHAPE;
    if (s->stride[3] != 1 || s->stride[2] != V || s->stride[1] != kK * V || s->stride[0] != HV * kK * V || !aligned16(s->data))
      return FLA_ERR_LAYOUT;
  }
  if ((st = kda_check_rstd(a->q_rstd, a->k_rstd, B, T, HK))) return st;
  if (a->chunk_size != kC) return FLA_ERR_VALUE;
  uint64_t off[4], off_saved, so[5], fo[5];
  const bool have_saved = a->saved.data != nullptr;
  const SegPlan plan = kda_bwd_plan(a, total_chunks, N);
  const uint64_t need = kda_bwd_ws_layout(total_chunks, HV, nvb, B * T, have_saved, plan, &off_saved, off);
  if (!workspace || workspace_bytes < need || !aligned16(workspace)) return FLA_ERR_WORKSPACE;
  const uint64_t sbytes = kda_saved_layout(total_chunks, HV, nvb, B * T, plan.split ? plan.count : 0, so);
  if (have_saved && (a->saved.dtype != FLA_BF16 || a->saved.ndim != 1 || uint64_t(a->saved.shape[0]) * 2 < sbytes ||
                     !aligned16(a->saved.data)))
    return FLA_ERR_SHAPE;
  kda_ws_layout(total_chunks, HV, fo);

  uint8_t* ws = static_cast<uint8_t*>(workspace);
  uint8_t* sv = have_saved ? static_cast<uint8_t*>(a->saved.data) : ws + off_saved;
  uint8_t* fws = sv + so[0];
  KdaParams f{};
  f.q = static_cast<const bf16*>(a->q.data); f.k = static_cast<const bf16*>(a->k.data); f.v = static_cast<const bf16*>(a->v.data);
  f.g = a->g.data; f.beta = a->beta.data;
  f.gk_out = reinterpret_cast<float*>(sv + so[1]);
  f.status = reinterpret_cast<int*>(ws);
  f.qk_img = reinterpret_cast<bf16*>(fws + fo[0]); f.kn_img = reinterpret_cast<bf16*>(fws + fo[1]);
  f.p_img = reinterpret_cast<bf16*>(fws + fo[2]); f.x_img = reinterpret_cast<bf16*>(fws + fo[3]);
  f.vec = reinterpret_cast<float*>(fws + fo[4]);
  f.s_img = reinterpret_cast<bf16*>(sv + so[2]); f.vn_img = reinterpret_cast<bf16*>(sv + so[3]);
  f.h0 = static_cast<const float*>(a->initial_state.data);
  f.cu_seqlens = static_cast<const int32_t*>(a->cu_seqlens.data);
  f.chunk_offsets = static_cast<const int32_t*>(a->chunk_offsets.data);
  f.q_st = a->q.stride[1]; f.q_sh = a->q.stride[2]; f.k_st = a->k.stride[1]; f.k_sh = a->k.stride[2];
  f.v_st = a->v.stride[1]; f.v_sh = a->v.stride[2];
  f.g_st = a->g.stride[1]; f.g_sh = a->g.stride[2]; f.beta_st = a->beta.stride[1];
  f.N = N; f.T = int(T); f.HK = int(HK); f.HV = int(HV); f.total_tokens = B * T; f.V = int(V); f.nvb = int(nvb);
  f.g_is_f32 = a->g.dtype == FLA_F32; f.beta_is_f32 = a->beta.dtype == FLA_F32;
  f.gate_mode = 0; f.scale = a->scale;
  f.seg_len = plan.len; f.seg_m = reinterpret_cast<bf16*>(sv + so[4]); f.seg_h = reinterpret_cast<float*>(ws + off[3]);
  f.q_rstd = static_cast<float*>(a->q_rstd.data); f.k_rstd = static_cast<float*>(a->k_rstd.data);   // (written again by the recomputed forward)

  KdaBwdParams p{};
  p.q = f.q; p.k = f.k; p.q_rstd = f.q_rstd; p.k_rstd = f.k_rstd;
  p.q_st = f.q_st; p.q_sh = f.q_sh; p.k_st = f.k_st; p.k_sh = f.k_sh;
  p.v = f.v; p.dO = static_cast<const bf16*>(a->d_o.data); p.beta = a->beta.data;
  p.qk_img = f.qk_img; p.kn_img = f.kn_img; p.p_img = f.p_img; p.x_img = f.x_img; p.vec = f.vec; p.gk = f.gk_out;
  p.s_img = f.s_img; p.vn_img = f.vn_img;
  p.ds_img = reinterpret_cast<bf16*>(ws + off[0]); p.dz_img = reinterpret_cast<bf16*>(ws + off[1]);
  p.bz = reinterpret_cast<float*>(ws + off[2]);
  p.seg_len = plan.len; p.seg_m = f.seg_m; p.seg_dh = f.seg_h; p.clear = have_saved;
  p.dht = static_cast<const float*>(a->dht.data); p.dh0 = static_cast<float*>(a->dh0.data);
  p.dq = a->dq.data; p.dk = a->dk.data; p.dv = a->dv.data; p.dg = a->dg.data; p.dbeta = a->dbeta.data;
  p.cu_seqlens = f.cu_seqlens; p.chunk_offsets = f.chunk_offsets;
  p.v_st = f.v_st; p.v_sh = f.v_sh; p.do_st = a->d_o.stride[1]; p.do_sh = a->d_o.stride[2]; p.beta_st = f.beta_st;
  p.dq_st = a->dq.stride[1]; p.dq_sh = a->dq.stride[2]; p.dk_st = a->dk.stride[1]; p.dk_sh = a->dk.stride[2];
  p.dv_st = a->dv.stride[1]; p.dv_sh = a->dv.stride[2]; p.dg_st = a->dg.stride[1]; p.dg_sh = a->dg.stride[2];
  p.total_tokens = B * T; p.n1 = N;
  p.N = N; p.T = int(T); p.HK = int(HK); p.HV = int(HV); p.V = int(V); p.nvb = int(nvb);
  p.beta_is_f32 = f.beta_is_f32;
  p.dq_f32 = a->dq.dtype == FLA_F32; p.dk_f32 = a->dk.dtype == FLA_F32; p.dv_f32 = a->dv.dtype == FLA_F32;
  p.dg_f32 = a->dg.dtype == FLA_F32; p.dbeta_f32 = a->dbeta.dtype == FLA_F32;
  p.scale = a->scale;
  p.status = f.status;
  p.counter = f.status + 16;      // both inside the workspace's 256-byte head

  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  if (!have_saved && (st = kda_launch_forward(f, total_chunks, plan.count, cs))) return st;
  static std::atomic<bool> attr_done_dev[64] = {};   // per device ordinal; setting the attributes twice is harmless
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return FLA_ERR_CUDA;
  if (!attr_done_dev[dev]) {
    for (auto* scan : {kda_scan_bwd_kernel<false, false>, kda_scan_bwd_kernel<false, true>, kda_scan_bwd_kernel<true, true>})
      if (cudaFuncSetAttribute(scan, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kKdaScanBwdSmem) + 1024) != cudaSuccess) return FLA_ERR_CUDA;
    for (auto* par : {kda_bwd_par_kernel<2, false>, kda_bwd_par_kernel<4, false>, kda_bwd_par_kernel<2, true>, kda_bwd_par_kernel<4, true>})
      if (cudaFuncSetAttribute(par, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kKdaParSmem) + 1024) != cudaSuccess) return FLA_ERR_CUDA;
    attr_done_dev[dev] = true;
  }
  CUtensorMap tm_gk, tm_v, tm_d;
  if (make_row_tile_map(&tm_v, p.v, uint64_t(V), uint64_t(HV), uint64_t(B * T), uint64_t(p.v_sh), uint64_t(p.v_st)) ||
      make_row_tile_map(&tm_d, p.dO, uint64_t(V), uint64_t(HV), uint64_t(B * T), uint64_t(p.do_sh), uint64_t(p.do_st)))
    return FLA_ERR_CUDA;
  if (make_row_tile_map_f32(&tm_gk, p.gk, kK, uint64_t(HV), uint64_t(B * T), uint64_t(kK), uint64_t(HV) * kK)) return FLA_ERR_CUDA;
  // more scan chains (one CTA per SM each) than SMs: two halves of the batch on two streams, so that the chunk-parallel
  // kernel of the first half fills the SMs the second half's scan leaves idle (aux_stream.h)
  AuxStream* aux = nullptr;
  if (N >= 2 && !plan.split && HV * (V / 128) * N > sm_count(dev) && !kernel_timing_enabled()) aux = aux_stream_for(dev, cs);
  auto launch_scan = [&](const KdaBwdParams& pp, int64_t segments, cudaStream_t st_) {
    const dim3 grid(unsigned(HV * (V / 128)), unsigned(segments));
    if (plan.split) {
      const cudaError_t e = launch_after(!aux, kda_scan_bwd_kernel<true, true>, grid, kScanThreads, kKdaScanBwdSmem + 1024, st_, pp, tm_v, tm_d);
      if (e != cudaSuccess) return e;
    }
    return launch_after(!aux, plan.split ? kda_scan_bwd_kernel<false, true> : kda_scan_bwd_kernel<false, false>, grid, kScanThreads, kKdaScanBwdSmem + 1024, st_, pp,
                      tm_v, tm_d);
  };
  auto launch_par = [&](const KdaBwdParams& pp, int64_t chunks, cudaStream_t st_) {
    auto* par = nvb == 2 ? (pp.q_rstd ? kda_bwd_par_kernel<2, true> : kda_bwd_par_kernel<2, false>)
                         : (pp.q_rstd ? kda_bwd_par_kernel<4, true> : kda_bwd_par_kernel<4, false>);
    return launch_after(!aux, par, unsigned(std::min<int64_t>(chunks * HK, sm_count(dev))), kParThreads, kKdaParSmem + 1024, st_, pp, int(chunks), tm_gk);
  };
  if (aux) {
    std::lock_guard<std::mutex> lk(aux->mu);
    const int n1 = N / 2;
    KdaBwdParams p2 = p;
    p.n1 = p2.n0 = n1;
    p2.counter = p.counter + 16;
    if (cudaEventRecord(aux->fork, cs) != cudaSuccess || cudaStreamWaitEvent(aux->s, aux->fork, 0) != cudaSuccess) return FLA_ERR_CUDA;
    bool launched = launch_scan(p, n1, cs) == cudaSuccess && launch_scan(p2, N - n1, aux->s) == cudaSuccess;
    // a packed batch's halves hold chunk counts the host does not have: the kernel looks up its own
    const int64_t nt = (T + kC - 1) / kC;
    launched = launched && launch_par(p, p.cu_seqlens ? total_chunks : n1 * nt, cs) == cudaSuccess &&
               launch_par(p2, p.cu_seqlens ? total_chunks : (N - n1) * nt, aux->s) == cudaSuccess;
    if (cudaEventRecord(aux->join, aux->s) != cudaSuccess || cudaStreamWaitEvent(cs, aux->join, 0) != cudaSuccess) return FLA_ERR_CUDA;
    return launched ? FLA_OK : FLA_ERR_CUDA;
  }
  {
    KernelTimer kt("kda_bwd_dhu", cs);
    if (launch_scan(p, plan.count, cs) != cudaSuccess) return FLA_ERR_CUDA;
  }
  {
    KernelTimer kt("kda_bwd_par", cs);
    return cuda_status(launch_par(p, total_chunks, cs));
  }
}

