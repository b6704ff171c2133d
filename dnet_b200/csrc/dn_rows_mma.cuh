// dn_rows_mma.cuh -- weight-streaming products of a few rows (up to 8 NT tokens) on the tensor cores, bf16.  Both libraries use it.
//
// Bound by reading the weights once.  With fused multiply-adds every weight costs a conversion and one instruction a token: at four
// tokens an SM issued 118 instructions for a kilobyte of weights and the row kernels ran at 55 % of the copy bandwidth.  Now they reach
// 6.3 TB/s (four tokens, two matrices of 14,336 x 4,096: 37 us, before 63): 13 steps of three layers and the head 5.82 ms -> 3.31.  Here a kilobyte
// (16 rows x 32 columns) takes three 16-byte loads a lane and two mma.sync m16n8k16: A = weights straight from global memory, B = the
// tokens (columns 0 .. N - 1, the rest zero), fp32 accumulators.  The columns of a product may be summed in any order as long as A and
// B agree, so lane (g, t) takes 8 neighbouring columns 8 t .. of weight rows g and g + 8 and of token g: they are the fragments of two
// MMAs as they lie.  (tcgen05 needs its operands in shared memory, 128 rows at a time: a few thousand features would fill a few SMs.)
// Every MMA starts from zero, and the sums of 16 products meet in ordinary fp32 additions, in pairs: handed on from MMA to MMA the
// accumulator is cut off, not rounded, at each step (4,096 columns: 4.7e-7 of the result against 64 bits; so 0.85e-7; a chain of multiply-adds
// a lane 0.9e-7).
// A block of eight warps takes 16 or 32 rows; each warp a share of the columns, the sums meet in shared memory in pairs of warps.
// The order of a token's sums depends on the sizes of the matrix alone.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

#include <type_traits>

namespace dn {

constexpr int RM_WARPS = 8, RM_THREADS = RM_WARPS * 32;
// Blocks of one tile: eight blocks of 32 columns in flight a warp and two thread blocks an SM, or four and three.  Two are the faster ones where
// all thread blocks run at once or in many waves (4,096 x 4,096, 4 tokens: 8.4 us against 8.7; x 14,336: 22.3 / 22.6; 14,336 x 4,096: 20.9 /
// 22.6), three where only they hold all (6,144 x 4,096: 12.4 / 10.9; 5,120 x 27,648: 58.6 / 46.2).  16 tokens: 4,096 x 14,336 26.6 / 34.9.
static inline bool rows_mma_deep(int blocks, int sms) { return blocks <= 2 * sms || blocks > 3 * sms; }
// Features from which a block takes two tiles (each token row is read for twice the weights): tiles of one fill three blocks an SM either way.
static inline bool rows_mma_wide(int features, int sms) { return features >= 3 * 16 * sms; }
// columns a lane loads at once: 16-byte rows of both operands
static inline bool rows_mma_ok(int K, const void* X, const void* W, const void* W2) {
  return K % 32 == 0 && ((((uintptr_t)X | (uintptr_t)W | (uintptr_t)(W2 ? W2 : W)) & 15) == 0);
}
__device__ __forceinline__ uint4 rm_ld_weights(const __nv_bfloat16* p) {
  uint4 r;
  asm volatile("ld.global.nc.L1::no_allocate.L2::256B.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
  return r;
}
__device__ __forceinline__ void rm_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
// 16 rows x 32 columns x 8 tokens
__device__ __forceinline__ void rm_mma32(float (&d)[4], const uint4& a, const uint4& b, const uint4& x) {
  float e[4];
  rm_mma(d, a.x, b.x, a.y, b.y, x.x, x.y);
  rm_mma(e, a.z, b.z, a.w, b.w, x.z, x.w);
#pragma unroll
  for (int i = 0; i < 4; ++i) d[i] += e[i];
}
// One warp's share of TILES tiles of 16 rows for NT groups of 8 tokens.  w: the matrices' rows 0 (row pitch K), r0: a tile's first row,
// rows: how many the matrix has (rows past it are read again and dropped by the caller); X [N][K]; columns 32 kb0 .. 32 kb1.
// U: blocks of 32 columns with all their loads in flight.  ready(): called once the first weights are on their way and before the first row is read.  acc: rows g, g + 8 x tokens 2 t, 2 t + 1
struct RmNow { __device__ __forceinline__ void operator()() const {} };
template <int TILES, int NT, int U, class Ready>
__device__ __forceinline__ void rows_mma(const __nv_bfloat16* const (&w)[TILES], const int (&r0)[TILES], int rows, const __nv_bfloat16* X, int N, int K, int kb0,
                                         int kb1, float (&acc)[TILES][NT][4], Ready ready) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const __nv_bfloat16 *wa[TILES], *wb[TILES], *x[NT];
  bool live[NT];
#pragma unroll
  for (int i = 0; i < TILES; ++i) {
#pragma unroll
    for (int q = 0; q < NT; ++q) acc[i][q][0] = acc[i][q][1] = acc[i][q][2] = acc[i][q][3] = 0.f;
    wa[i] = w[i] + (size_t)min(r0[i] + g, rows - 1) * K + 8 * t;
    wb[i] = w[i] + (size_t)min(r0[i] + g + 8, rows - 1) * K + 8 * t;
  }
#pragma unroll
  for (int q = 0; q < NT; ++q) {
    live[q] = 8 * q + g < N;
    x[q] = X + (size_t)(live[q] ? 8 * q + g : 0) * K + 8 * t;
  }
  // n blocks at once (compile time: a run-time bound would put a branch between the loads); wait: call ready() behind the weights' loads
  auto go = [&](auto nc, int kb, bool wait) {
    constexpr int n = decltype(nc)::value;
    uint4 a[n][TILES], b[n][TILES], xv[n][NT];
#pragma unroll
    for (int u = 0; u < n; ++u)
#pragma unroll
      for (int i = 0; i < TILES; ++i) { a[u][i] = rm_ld_weights(wa[i] + (kb + u) * 32); b[u][i] = rm_ld_weights(wb[i] + (kb + u) * 32); }
    if (wait) ready();
#pragma unroll
    for (int u = 0; u < n; ++u)
#pragma unroll
      for (int q = 0; q < NT; ++q) xv[u][q] = live[q] ? *reinterpret_cast<const uint4*>(x[q] + (kb + u) * 32) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int u = 0; u < n; u += 2)
#pragma unroll
      for (int i = 0; i < TILES; ++i)
#pragma unroll
        for (int q = 0; q < NT; ++q) {
          float d[4], e[4];
          rm_mma32(d, a[u][i], b[u][i], xv[u][q]);
          if constexpr (n > 1) {
            rm_mma32(e, a[u + 1][i], b[u + 1][i], xv[u + 1][q]);
#pragma unroll
            for (int k = 0; k < 4; ++k) d[k] += e[k];
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) acc[i][q][k] += d[k];
        }
  };
  int kb = kb0;
  if (kb + U <= kb1) { go(std::integral_constant<int, U>{}, kb, true); kb += U; }
  else ready();
#pragma unroll 1
  for (; kb + U <= kb1; kb += U) go(std::integral_constant<int, U>{}, kb, false);
  if (U > 4 && kb + 4 <= kb1) { go(std::integral_constant<int, 4>{}, kb, false); kb += 4; }
  if (kb + 2 <= kb1) { go(std::integral_constant<int, 2>{}, kb, false); kb += 2; }
  if (kb < kb1) go(std::integral_constant<int, 1>{}, kb, false);
}
// A block's tiles: every warp its share of the columns, then the sums of the eight.  red: [RM_WARPS][TILES][NT][16 rows][8 tokens] floats
template <int TILES, int NT = 1, int U = 4, class Ready = RmNow>
__device__ __forceinline__ void rows_mma_block(const __nv_bfloat16* const (&w)[TILES], const int (&r0)[TILES], int rows, const __nv_bfloat16* X, int N, int K,
                                               float* red, Ready ready = Ready()) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nb = K / 32;
  float acc[TILES][NT][4];
  rows_mma<TILES, NT, U>(w, r0, rows, X, N, K, nb * warp / RM_WARPS, nb * (warp + 1) / RM_WARPS, acc, ready);
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int i = 0; i < TILES; ++i)
#pragma unroll
    for (int q = 0; q < NT; ++q) {
      float* r = red + ((warp * TILES + i) * NT + q) * 128;
      *reinterpret_cast<float2*>(r + g * 8 + 2 * t) = make_float2(acc[i][q][0], acc[i][q][1]);
      *reinterpret_cast<float2*>(r + (g + 8) * 8 + 2 * t) = make_float2(acc[i][q][2], acc[i][q][3]);
    }
  __syncthreads();
}
// (row, token) `at` = row * 8 + token of tile i's group q
template <int TILES, int NT = 1>
__device__ __forceinline__ float rows_mma_sum(const float* red, int i, int at, int q = 0) {
  float v[RM_WARPS];
#pragma unroll
  for (int k = 0; k < RM_WARPS; ++k) v[k] = red[((k * TILES + i) * NT + q) * 128 + at];
  return ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
}

}  // namespace dn
