// dn_rows_mma.cuh -- weight-streaming products of a few rows (up to 8 tokens) on the tensor cores, bf16.  Both libraries use it.
//
// Bound by reading the weights once.  With fused multiply-adds every weight costs a conversion and one instruction a token: at four
// tokens an SM issued 118 instructions for a kilobyte of weights and the row kernels ran at 55 % of the copy bandwidth.  Now they reach
// 6.3 TB/s (four tokens, two matrices of 14,336 x 4,096: 37 us, before 63): 13 steps of three layers and the head 5.82 ms -> 3.31.  Here a kilobyte
// (16 rows x 32 columns) takes three 16-byte loads a lane and two mma.sync m16n8k16: A = weights straight from global memory, B = the
// tokens (columns 0 .. N - 1, the rest zero), fp32 accumulators.  The columns of a product may be summed in any order as long as A and
// B agree, so lane (g, t) takes 8 neighbouring columns 8 t .. of weight rows g and g + 8 and of token g: they are the fragments of two
// MMAs as they lie.  (tcgen05 needs its operands in shared memory, 128 rows at a time: a few thousand features would fill a few SMs.)
// A block of eight warps takes 16 or 32 rows; each warp a share of the columns, the sums meet in shared memory in the order of the warps.
// The order of a token's sums depends on the sizes of the matrix alone.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

namespace dn {

constexpr int RM_WARPS = 8, RM_THREADS = RM_WARPS * 32;
// columns a lane loads at once: 16-byte rows of both operands
static inline bool rows_mma_ok(int K, const void* X, const void* W, const void* W2) {
  return K % 32 == 0 && ((((uintptr_t)X | (uintptr_t)W | (uintptr_t)(W2 ? W2 : W)) & 15) == 0);
}
__device__ __forceinline__ uint4 rm_ld_weights(const __nv_bfloat16* p) {
  uint4 r;
  asm volatile("ld.global.nc.L1::no_allocate.L2::256B.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
  return r;
}
__device__ __forceinline__ void rm_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// One warp's share of TILES tiles of 16 rows.  w: the matrices' rows 0 (row pitch K), r0: a tile's first row, rows: how many the matrix has
// (rows past it are read again and dropped by the caller); X [N][K]; columns 32 kb0 .. 32 kb1.  acc: rows g, g + 8 x tokens 2 t, 2 t + 1
template <int TILES>
__device__ __forceinline__ void rows_mma(const __nv_bfloat16* const (&w)[TILES], const int (&r0)[TILES], int rows, const __nv_bfloat16* X, int N, int K, int kb0,
                                         int kb1, float (&acc)[TILES][4]) {
  constexpr int U = TILES == 1 ? 8 : 4;      // blocks of 32 columns with all their loads in flight
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const __nv_bfloat16 *wa[TILES], *wb[TILES];
#pragma unroll
  for (int i = 0; i < TILES; ++i) {
    acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    wa[i] = w[i] + (size_t)min(r0[i] + g, rows - 1) * K + 8 * t;
    wb[i] = w[i] + (size_t)min(r0[i] + g + 8, rows - 1) * K + 8 * t;
  }
  const bool live = g < N;
  const __nv_bfloat16* x = X + (size_t)(live ? g : 0) * K + 8 * t;
  auto go = [&](int kb, int n) {
    uint4 a[U][TILES], b[U][TILES], xv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u >= n) break;
      const int k = (kb + u) * 32;
#pragma unroll
      for (int i = 0; i < TILES; ++i) { a[u][i] = rm_ld_weights(wa[i] + k); b[u][i] = rm_ld_weights(wb[i] + k); }
      xv[u] = live ? *reinterpret_cast<const uint4*>(x + k) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u >= n) break;
#pragma unroll
      for (int i = 0; i < TILES; ++i) {
        rm_mma(acc[i], a[u][i].x, b[u][i].x, a[u][i].y, b[u][i].y, xv[u].x, xv[u].y);
        rm_mma(acc[i], a[u][i].z, b[u][i].z, a[u][i].w, b[u][i].w, xv[u].z, xv[u].w);
      }
    }
  };
  int kb = kb0;
#pragma unroll 1
  for (; kb + U <= kb1; kb += U) go(kb, U);
#pragma unroll 1
  for (; kb < kb1; ++kb) go(kb, 1);
}
// A block's tiles: every warp its share of the columns, then the sums of the eight.  red: [RM_WARPS][TILES][16 rows][8 tokens] floats
template <int TILES>
__device__ __forceinline__ void rows_mma_block(const __nv_bfloat16* const (&w)[TILES], const int (&r0)[TILES], int rows, const __nv_bfloat16* X, int N, int K,
                                               float* red) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nb = K / 32;
  float acc[TILES][4];
  rows_mma<TILES>(w, r0, rows, X, N, K, nb * warp / RM_WARPS, nb * (warp + 1) / RM_WARPS, acc);
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int i = 0; i < TILES; ++i) {
    float* r = red + (warp * TILES + i) * 128;
    *reinterpret_cast<float2*>(r + g * 8 + 2 * t) = make_float2(acc[i][0], acc[i][1]);
    *reinterpret_cast<float2*>(r + (g + 8) * 8 + 2 * t) = make_float2(acc[i][2], acc[i][3]);
  }
  __syncthreads();
}
// (row, token) `at` = row * 8 + token of tile i
template <int TILES>
__device__ __forceinline__ float rows_mma_sum(const float* red, int i, int at) {
  float v = 0.f;
#pragma unroll
  for (int q = 0; q < RM_WARPS; ++q) v += red[(q * TILES + i) * 128 + at];
  return v;
}

}  // namespace dn
