// Inverse of a 64 x 64 unit lower-triangular matrix  X = (I + A)^-1,  A strictly lower triangular, fp32, in shared memory: the
// last step of the GDN and KDA prep kernels (the reference's solve_tri operator,
// fla/ops/ascendc/gdn/chunk_gdn_fwd/solve_tri/README.md:9-13, which inverts in bf16 on the matrix unit; here the inverse is
// fp32 throughout and rounded to bf16 value + residual once at the end).
//
// Four or eight warps take one matrix.  Forward substitution over all 64 rows is a chain of 64 dependent steps; by blocks it is 16: the
// four 16 x 16 diagonal blocks are substituted side by side (a thread per column, its 16 entries in registers), then
//     X_BL = -X_22 (A_BL X_11)
// fills the block below the diagonal, for the two 32 x 32 halves at once and then for the whole matrix.  Those products are
// register tiles (2 to 8 entries per thread) whose operands are read as 16-byte pieces: the matrix is kept transposed,
// AT[j][i] = A[i][j], which gives a thread's four rows of the left factor in one piece and four steps of the reduction of the right
// factor in another.
// The stand-alone kernel this replaces (one thread per column, 64 dependent steps, A read from and X written to memory) took
// 152 us for 16,384 matrices, on top of the 185 us of the GDN prep kernel that made them.
#pragma once
#include "gdn_common.cuh"

namespace fla {

constexpr int kTriStride = 68;                      // fp32 row stride: 16-byte aligned rows that spread over the banks
constexpr int kTriTile = kC * kTriStride;           // floats per matrix

template <int THREADS>
__device__ __forceinline__ void tri_sync(int bar) { asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(THREADS) : "memory"); }

// acc[cc][r] = sum_k L[r][k] R[k][c + 8 cc] over k0 <= k < k1, L at left[k][r] (NR rows), R at right[8 cc][k] (transposed storage;
// columns 8 apart so that eight lanes with neighbouring columns read 16-byte pieces from all banks)
template <int NC, int NR>
__device__ __forceinline__ void tri_product(const float* left, const float* right, int k0, int k1, float (&acc)[NC][NR]) {
#pragma unroll
  for (int cc = 0; cc < NC; ++cc)
#pragma unroll
    for (int r = 0; r < NR; ++r) acc[cc][r] = 0.f;
#pragma unroll 2
  for (int k = k0; k < k1; k += 4) {
    float rv[NC][4];
#pragma unroll
    for (int cc = 0; cc < NC; ++cc) {
      const float4 x = *reinterpret_cast<const float4*>(right + cc * 8 * kTriStride + k);
      rv[cc][0] = x.x; rv[cc][1] = x.y; rv[cc][2] = x.z; rv[cc][3] = x.w;
    }
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      float l[NR];
      if constexpr (NR == 4) {
        const float4 x = *reinterpret_cast<const float4*>(left + (k + kk) * kTriStride);
        l[0] = x.x; l[1] = x.y; l[2] = x.z; l[3] = x.w;
      } else {
        const float2 x = *reinterpret_cast<const float2*>(left + (k + kk) * kTriStride);
        l[0] = x.x; l[1] = x.y;
      }
#pragma unroll
      for (int cc = 0; cc < NC; ++cc)
#pragma unroll
        for (int r = 0; r < NR; ++r) acc[cc][r] += l[r] * rv[cc][kk];
    }
  }
}

// NR consecutive entries of one column, times sign
template <int NR>
__device__ __forceinline__ void tri_put(float* dst, const float (&x)[NR], float sign) {
  if constexpr (NR == 4) *reinterpret_cast<float4*>(dst) = make_float4(sign * x[0], sign * x[1], sign * x[2], sign * x[3]);
  else *reinterpret_cast<float2*>(dst) = make_float2(sign * x[0], sign * x[1]);
}

// In place: AT becomes X^T.  Only the 16 x 16 diagonal blocks and what lies below them (i > j) are read, the entries of the diagonal
// blocks with i <= j must be zero; the blocks above the diagonal take the intermediate products and hold no zeros afterwards
// (tri_store_* know).  Called by THREADS (128 or 256) threads, t = 0 .. THREADS - 1, that share named barrier `bar`; the matrix
// must be visible to all of them before, and the inverse is after.
template <int THREADS>
__device__ __forceinline__ void tri_invert(float* AT, int t, int bar) {
  if (t < 64) {      // diagonal blocks: column c of block b; the sixteen lanes of a block are in one warp
    const int b = (t >> 4) * 16, c = t & 15;
    const float* blk = AT + b * kTriStride + b;
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = i == c ? 1.f : 0.f;
#pragma unroll
    for (int j = 0; j < 15; ++j) {
#pragma unroll
      for (int i4 = (j + 1) & ~3; i4 < 16; i4 += 4) {
        const float4 a = *reinterpret_cast<const float4*>(blk + j * kTriStride + i4);   // zero for i <= j
        x[i4] -= a.x * x[j]; x[i4 + 1] -= a.y * x[j]; x[i4 + 2] -= a.z * x[j]; x[i4 + 3] -= a.w * x[j];
      }
    }
    __syncwarp();
    float* dst = AT + (b + c) * kTriStride + b;
#pragma unroll
    for (int i = 0; i < 16; i += 4) *reinterpret_cast<float4*>(dst + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
  }
  tri_sync<THREADS>(bar);
  {                  // 16 x 16 blocks below the diagonal of the two 32 x 32 halves: 512 outputs
    constexpr int NR = 512 / THREADS;
    const int u = t % (THREADS / 2), b = t / (THREADS / 2) * 32, c = u & 15, r = (u >> 4) * NR;
    float acc[1][NR];
    tri_product<1, NR>(AT + b * kTriStride + b + 16 + r, AT + (b + c) * kTriStride + b, 0, 16, acc);
    float* tmp = AT + (b + 16 + c) * kTriStride + b;         // the block above the diagonal
    tri_put(tmp + r, acc[0], 1.f);
    tri_sync<THREADS>(bar);
    tri_product<1, NR>(AT + (b + 16) * kTriStride + b + 16 + r, tmp, 0, 16, acc);
    tri_put(AT + (b + c) * kTriStride + b + 16 + r, acc[0], -1.f);
    tri_sync<THREADS>(bar);
  }
  {                  // the 32 x 32 block below the diagonal: a warp stays within one 16 x 16 quarter, so that it can skip the half of
                     // the reduction that meets the zeros of X_11 (columns 16..31) or of X_22 (rows 0..15)
    constexpr int NC = 256 / THREADS, NL = 16 / NC;          // columns per thread, 8 apart; lanes side by side in a column group
    const int u = t % (THREADS / 4), cq = t / (THREADS / 2), rq = t / (THREADS / 4) & 1;
    const int c = cq * 16 + u % NL, r = rq * 16 + u / NL * 4;
    float acc[NC][4];
    tri_product<NC, 4>(AT + 32 + r, AT + c * kTriStride, cq * 16, 32, acc);
    float* tmp = AT + (32 + c) * kTriStride;
#pragma unroll
    for (int cc = 0; cc < NC; ++cc) tri_put(tmp + cc * 8 * kTriStride + r, acc[cc], 1.f);
    tri_sync<THREADS>(bar);
    tri_product<NC, 4>(AT + 32 * kTriStride + 32 + r, tmp, 0, 16 + rq * 16, acc);
#pragma unroll
    for (int cc = 0; cc < NC; ++cc) tri_put(AT + (c + cc * 8) * kTriStride + 32 + r, acc[cc], -1.f);
    tri_sync<THREADS>(bar);
  }
}

// X (value + residual) to memory; rows past the end of the sequence as zeros.
// Strips of 8 rows, [value | residual][8 strips][64 columns][16 bytes]: a piece is 8 consecutive entries of a row of X^T.
template <int THREADS>
__device__ __forceinline__ void tri_store_strips(const float* XT, uint8_t* img, int rows, int t) {
#pragma unroll
  for (int q = 0; q < 512 / THREADS; ++q) {
    const int idx = t + q * THREADS, g = idx >> 6, c = idx & 63;
    const float4 a = *reinterpret_cast<const float4*>(XT + c * kTriStride + g * 8), b = *reinterpret_cast<const float4*>(XT + c * kTriStride + g * 8 + 4);
    float x[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    const int lim = (g >> 1) < (c >> 4) ? 0 : rows;      // blocks above the diagonal are zero
    if (lim < kC) {
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = g * 8 + i < lim ? x[i] : 0.f;
    }
    uint4 hi, lo;
    split8(x, hi, lo);
    *reinterpret_cast<uint4*>(img + idx * 16) = hi;
    *reinterpret_cast<uint4*>(img + 8192 + idx * 16) = lo;
  }
}

// The swizzled 64 x 64 operand panels (sm100.cuh), value then residual.
template <int THREADS>
__device__ __forceinline__ void tri_store_panels(const float* XT, uint8_t* img, int rows, int t) {
#pragma unroll
  for (int q = 0; q < 512 / THREADS; ++q) {
    const int idx = t + q * THREADS, i = idx & 63, ch = idx >> 6;
    float x[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = i < rows && (i >> 4) >= (ch >> 1) ? XT[(ch * 8 + j) * kTriStride + i] : 0.f;
    uint4 hi, lo;
    split8(x, hi, lo);
    const uint32_t off = panel_chunk_off(i, ch);
    *reinterpret_cast<uint4*>(img + off) = hi;
    *reinterpret_cast<uint4*>(img + 8192 + off) = lo;
  }
}

}  // namespace fla
