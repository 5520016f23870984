// Splitting a long chain over several SMs.
//
// A scan visits the chunks of one (sequence, value head) one after the other on one SM; with few sequences and heads most SMs
// stay idle for the whole call (a single 16,384-token prompt with 32 heads: 32 chains of 256 chunks on 148 SMs).  The state update of a
// chunk is linear in the state, S' = M_c S + H_c, so a run of chunks (a segment) is S_end = M S_start + H as well, and
//   1. a state-only pass over each segment gives H (from the zero state; the first segment from the true one) and M (the same
//      pass with zero values, from the identity: its 128 columns take the place of the value channels) - all segments at once;
//   2. the full scan runs all segments at once; a segment's CTA first walks S <- M_i S + H_i over the segments before it, one
//      128 x 128 x 128 product each (bf16 value + residual in three passes, fp32 accumulation, like every product of the scan).
// The reverse scan's gradient is carried by the transpose of the same M.
#pragma once
#include "gdn_common.cuh"
#include "aux_stream.h"

namespace fla {

constexpr int kWholeSequence = 1 << 30;      // as a segment length: chains are not split
struct SegPos {
  SeqInfo sq;       // the sequence from the segment's first chunk on (bos, len, cbase), so that chunks count from there
  int n, s, ns;     // sequence, segment inside it, segments of the sequence
  int nt;           // chunks of the segment
};
// Called by whole warps: the sequence of [first, first + count) with the `place`-th most chunks.  Whole chains start in this order: hardware hands
// out CTAs in order, and a long chain that starts last is what all other SMs wait for (22 prompts x 32 heads, 11,003 tokens: 282 -> 240 us).
__device__ __forceinline__ int by_length(const int32_t* chunk_offsets, int first, int count, int place) {
  const int lane = threadIdx.x & 31;
  int nt[2], rank[2] = {0, 0};
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int n = lane + i * 32;
    nt[i] = n < count ? chunk_offsets[first + n + 1] - chunk_offsets[first + n] : -1;
  }
  for (int j = 0; j < count; ++j) {
    const int other = __shfl_sync(0xffffffffu, j < 32 ? nt[0] : nt[1], j & 31);
#pragma unroll
    for (int i = 0; i < 2; ++i) rank[i] += other > nt[i] || (other == nt[i] && j < lane + i * 32);
  }
  const unsigned lo = __ballot_sync(0xffffffffu, nt[0] >= 0 && rank[0] == place), hi = __ballot_sync(0xffffffffu, nt[1] >= 0 && rank[1] == place);
  return first + (lo ? __ffs(lo) - 1 : hi ? 31 + __ffs(hi) : place);
}
constexpr int kMostByLength = 64;      // sequences that are put in order
// Called by whole warps: segment `flat` of the batch; false past the last one (packed batches launch an upper bound).  [n0, n1): the sequences of
// this launch.
template <bool kSplit>
__device__ __forceinline__ bool segment_pos(const int32_t* cu_seqlens, const int32_t* chunk_offsets, int N, int T, int seg_len, int flat, SegPos& r, int n0, int n1) {
  if (!kSplit) {
    r.n = cu_seqlens && n1 - n0 <= kMostByLength ? by_length(chunk_offsets, n0, n1 - n0, flat - n0) : flat;
    r.s = 0;
    r.ns = 1;
  } else if (!cu_seqlens) {
    const int nt = (T + kC - 1) / kC, ns = max(1, (nt + seg_len - 1) / seg_len);
    r.n = flat / ns;
    r.s = flat - r.n * ns;
    r.ns = ns;
  } else {
    const int lane = threadIdx.x & 31;
    int base = 0, i0 = 0;
    for (; i0 < N; i0 += 32) {
      const int i = i0 + lane;
      const int own = i < N ? max(1, (chunk_offsets[i + 1] - chunk_offsets[i] + seg_len - 1) / seg_len) : 0;
      int incl = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
      }
      const unsigned past = __ballot_sync(0xffffffffu, base + incl > flat);
      if (past) {
        const int k = __ffs(past) - 1;
        r.n = i0 + k;
        r.ns = __shfl_sync(0xffffffffu, own, k);
        r.s = flat - base - (__shfl_sync(0xffffffffu, incl, k) - r.ns);
        break;
      }
      base += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (i0 >= N) return false;
  }
  r.sq = seq_info(cu_seqlens, chunk_offsets, r.n, T);
  r.nt = r.sq.nt;
  if (kSplit && r.ns > 1) {
    const int c0 = r.s * seg_len;
    r.nt = min(seg_len, r.sq.nt - c0);
    r.sq.bos += c0 * kC;
    r.sq.len -= c0 * kC;
    r.sq.cbase += c0;
  }
  return true;
}

// bytes of one (segment, value head): M as a value + residual image; H in fp32 per 128 value channels
constexpr uint64_t kSegMBytes = 65536, kSegHBytes = 65536;
// ---- host side
struct SegPlan {
  int len = kWholeSequence; // chunks per segment
  int64_t count = 0;        // segments of the batch (packed: an upper bound)
  bool split = false;
};
// Chooses the segment length by the time of the longest SM, in units of one full chunk step (3.2 to 3.6 us).  `state` is the cost of a
// state-only step; a product of the start-up walk costs about half a step, a pass of its own (launch, start-up) about three.  heads: CTAs per segment of the full scan; m_heads: matrices M per segment.  Splitting has to win a
// tenth to be taken.
inline SegPlan plan_segments(int64_t N, int64_t total_chunks, int64_t max_nt, bool packed, int64_t heads, int64_t m_heads, double state,
                             int sms) {
  SegPlan best;
  best.count = N;
  auto waves = [&](double jobs) { return packed ? (jobs <= sms ? 1.0 : jobs / sms + 0.5) : double(int64_t((jobs + sms - 1) / sms)); };
  double t_best = 0.9 * (packed ? (N * heads <= sms ? double(max_nt) : double(total_chunks) * heads / sms + 0.5 * max_nt) : waves(double(N * heads)) * max_nt);
  for (int64_t S = 2; S <= 40 && S * 2 <= max_nt; ++S) {
    const int64_t len = (max_nt + S - 1) / S;
    const double segs = packed ? double(total_chunks) / len + N : double(N * S), cut = packed ? double(total_chunks) / len : double(N * (S - 1));
    const double jobs1 = cut * heads + (cut - (packed ? 0 : N)) * m_heads;
    const double t = waves(jobs1) * len * state + waves(segs * heads) * len + 0.5 * double(S - 2) + 3.0;
    if (t < t_best) {
      t_best = t;
      best.split = true;
      best.len = int(len);
      best.count = packed ? total_chunks / len + N : N * ((max_nt + len - 1) / len);
    }
  }
  return best;
}
// How the scans of one call split their chains: the same in its forward and its backward.  A state-only step takes as long as a full one
// (the outputs and score products it leaves out are off the chain).
inline SegPlan scan_plan(int64_t N, int64_t total_chunks, int64_t max_len, bool packed, int64_t HV, int64_t V) {
  return plan_segments(N, total_chunks, (max_len + kC - 1) / kC, packed, HV * (V / 128), HV, 1.0, current_sm_count());
}

}  // namespace fla
