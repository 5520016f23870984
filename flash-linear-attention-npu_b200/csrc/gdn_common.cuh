// Shared pieces of the chunked GDN kernels: parameter block, sequence/chunk geometry and small
// row-wise helpers for moving fp32 accumulator rows between TMEM, registers and operand panels.
#pragma once
#include "common/pdl.cuh"
#include <cuda_fp16.h>
#include "common/sm100.cuh"

namespace fla {

using bf16 = __nv_bfloat16;

constexpr int kC = 64;     // chunk length (tokens)
constexpr int kK = 128;    // key head dim
constexpr int kV = 128;    // value head dim
constexpr int kBV = 64;    // value columns owned by one CTA of the sequential kernels

struct SeqInfo {
  int bos;   // first token (flat index) of the sequence
  int len;   // tokens in the sequence
  int nt;    // chunks in the sequence
  int cbase; // flat index of the sequence's first chunk (for per-chunk saved tensors)
};

// cu_seqlens == nullptr: sequence n is batch row n with T tokens.
__device__ __forceinline__ SeqInfo seq_info(const int32_t* cu_seqlens, const int32_t* chunk_offsets, int n, int T) {
  SeqInfo s;
  if (cu_seqlens) {
    s.bos = cu_seqlens[n];
    s.len = cu_seqlens[n + 1] - s.bos;
    s.cbase = chunk_offsets[n];
  } else {
    s.bos = n * T;
    s.len = T;
    s.cbase = n * ((T + kC - 1) / kC);
  }
  s.nt = (s.len + kC - 1) / kC;
  return s;
}

// The chunk-parallel kernels launch one CTA (per head) for each chunk there is, numbered through all sequences: a grid of
// (longest sequence) x (sequences) leaves most of a packed batch's CTAs with nothing to do (22 prompts of 11,003 tokens: 172 chunks, 1,034
// CTAs per head, 178 us for the GDN prep kernel where the chunks alone take 120).
struct ChunkPos {
  SeqInfo sq;
  int n, c;  // sequence, chunk inside it
};
// Called by whole warps.  `chunk` counts from the first chunk of sequence n0 (fixed lengths; packed: of the batch).
__device__ __forceinline__ ChunkPos chunk_pos(const int32_t* cu_seqlens, const int32_t* chunk_offsets, int N, int T, int n0, int chunk) {
  ChunkPos r;
  if (!cu_seqlens) {
    const int nt = (T + kC - 1) / kC, k = chunk / nt;
    r.n = n0 + k;
    r.sq = seq_info(nullptr, nullptr, r.n, T);
    r.c = chunk - k * nt;
    return r;
  }
  // the last sequence that starts at or before the chunk: 32 candidates at a time
  int lo = 0, n = N;
  const int lane = threadIdx.x & 31;
  while (n > 1) {
    const int step = (n + 31) / 32, i = lane * step;
    const unsigned le = __ballot_sync(0xffffffffu, i < n && chunk_offsets[lo + i] <= chunk);
    const int k = __popc(le) - 1;
    lo += k * step;
    n = min(step, n - k * step);
  }
  r.n = lo;
  r.sq = seq_info(cu_seqlens, chunk_offsets, lo, T);
  r.c = chunk - r.sq.cbase;
  return r;
}

__device__ __forceinline__ float ld_scalar(const void* p, int64_t idx, int is_f32) {
  return is_f32 ? static_cast<const float*>(p)[idx] : __bfloat162float(static_cast<const bf16*>(p)[idx]);
}

constexpr float kLog2e = 1.4426950408889634f;
// 2^x in one instruction (results below the normal range are zero): decays of arguments already scaled by log2(e)
__device__ __forceinline__ float exp2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Eight consecutive floats, 16-byte aligned.
__device__ __forceinline__ void gather8(const float* p, float* f) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}

// Load 64 consecutive fp32 accumulator columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld_row64(uint32_t taddr, float* v) {
  tmem_ld32(taddr, v);
  tmem_ld32(taddr + 32, v + 32);
  tmem_ld_wait();
}
__device__ __forceinline__ void tmem_st_row64(uint32_t taddr, const float* v) {
  tmem_st16(taddr, v);
  tmem_st16(taddr + 16, v + 16);
  tmem_st16(taddr + 32, v + 32);
  tmem_st16(taddr + 48, v + 48);
  tmem_st_wait();
}

// Write a 64-wide fp32 row as bf16 hi / lo residual rows of two panels.
__device__ __forceinline__ void row64_to_hilo(uint8_t* pan_hi, uint8_t* pan_lo, int row, const float* x) {
#pragma unroll
  for (int ch = 0; ch < 8; ++ch) {
    uint4 hi, lo;
    split8(x + ch * 8, hi, lo);
    const uint32_t off = panel_chunk_off(row, ch);
    *reinterpret_cast<uint4*>(pan_hi + off) = hi;
    *reinterpret_cast<uint4*>(pan_lo + off) = lo;
  }
}
__device__ __forceinline__ void row64_to_bf16(uint8_t* pan, int row, const float* x) {
#pragma unroll
  for (int ch = 0; ch < 8; ++ch) *reinterpret_cast<uint4*>(pan + panel_chunk_off(row, ch)) = pack8(x + ch * 8);
}

__device__ __forceinline__ void unpack_bf16x8(const uint4& raw, float* f) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __low2float(h[i]);
    f[2 * i + 1] = __high2float(h[i]);
  }
}

// 32 consecutive fp32 accumulator columns of this thread's TMEM lane <-> registers / split bf16 panels.
__device__ __forceinline__ void tmem_ld_row32(uint32_t taddr, float* v) {
  tmem_ld32(taddr, v);
  tmem_ld_wait();
}
__device__ __forceinline__ void tmem_st_row32(uint32_t taddr, const float* v) {
  tmem_st16(taddr, v);
  tmem_st16(taddr + 16, v + 16);
  tmem_st_wait();
}
// columns [32*half, 32*half + 32) of `row`
__device__ __forceinline__ void row32_to_hilo(uint8_t* pan_hi, uint8_t* pan_lo, int row, int half, const float* x) {
#pragma unroll
  for (int ch = 0; ch < 4; ++ch) {
    uint4 hi, lo;
    split8(x + ch * 8, hi, lo);
    const uint32_t off = panel_chunk_off(row, half * 4 + ch);
    *reinterpret_cast<uint4*>(pan_hi + off) = hi;
    *reinterpret_cast<uint4*>(pan_lo + off) = lo;
  }
}


// columns [32*half, 32*half + 32) of `row` as fp16 (11-bit significand: enough for the state copy in one pass)
__device__ __forceinline__ void row32_to_f16(uint8_t* pan, int row, int half, const float* x) {
#pragma unroll
  for (int ch = 0; ch < 4; ++ch) {
    uint4 v;
    __half2* h = reinterpret_cast<__half2*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(x[ch * 8 + 2 * i], x[ch * 8 + 2 * i + 1]);
    *reinterpret_cast<uint4*>(pan + panel_chunk_off(row, half * 4 + ch)) = v;
  }
}
__device__ __forceinline__ void unpack_f16x8(const uint4& raw, float* f) {
  const __half2* h = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __half22float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}

// The first CTA of an operator's first kernel clears the status word (a memset of its own was a launch more per call).  A wait
// that runs out does so after millions of polls: long after that CTA, which is the first to be scheduled, has passed here.
__device__ __forceinline__ void clear_status(int* status, bool first) {
  if (first && status) *status = 0;
}

// A wait that gives up records the timeout once; afterwards the thread stops waiting so that the kernel
// still terminates quickly (its results are then invalid, which the status word tells the host).
__device__ __forceinline__ void wait_or_mark(uint64_t* bar, uint32_t& phase, bool& dead, int* status) {
  if (!dead && !mbar_wait(bar, phase, status, 8 /* FLA_ERR_TIMEOUT */)) dead = true;
  phase ^= 1;
}


}  // namespace fla
