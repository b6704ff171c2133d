// dn_moe.cuh -- routed experts on the grouped tcgen05 GEMM (dn_gemm_tc.cuh, GROUPED): the plan that sorts the (token, choice)
// pairs by expert into tiles of rows, and the gather of the tokens' rows in that order.  Both libraries use it.
#pragma once
#include <stdint.h>
#include "dn_pdl.cuh"

namespace dn {

// pairs sorted by expert: pos[p] = row of pair p, row_tok[row] = its token, and the table of tiles of `rows` rows
struct MoePlan {
  int32_t* pos;        // [P]
  int32_t* row_tok;    // [P]
  int32_t* tile_e;     // [max tiles]
  int32_t* tile_r0;
  int32_t* tile_rows;
  int32_t* n_tiles;    // [1]
};
// E: outputs of the router; experts from Ereal on are identity experts: their pairs get rows but no tiles
__global__ void __launch_bounds__(1024) k_moe_plan(const int32_t* __restrict__ idx, int P, int top, int E, int rows, MoePlan pl, int Ereal) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ int32_t cnt[];      // [E] counts, [E + 1] offsets
  int32_t* off = cnt + E;
  for (int e = threadIdx.x; e < E; e += blockDim.x) cnt[e] = 0;
  __syncthreads();
  for (int p = threadIdx.x; p < P; p += blockDim.x) pl.pos[p] = atomicAdd(&cnt[idx[p]], 1);     // rank among its expert's pairs
  __syncthreads();
  if (threadIdx.x == 0) {
    int a = 0, t = 0;
    for (int e = 0; e < E; e++) {
      off[e] = a;
      for (int r = 0; e < Ereal && r < cnt[e]; r += rows, t++) {
        pl.tile_e[t] = e;
        pl.tile_r0[t] = a + r;
        pl.tile_rows[t] = min(rows, cnt[e] - r);
      }
      a += cnt[e];
    }
    *pl.n_tiles = t;
  }
  __syncthreads();
  for (int p = threadIdx.x; p < P; p += blockDim.x) {
    const int row = off[idx[p]] + pl.pos[p];
    pl.pos[p] = row;
    pl.row_tok[row] = p / top;
  }
}

// the tokens' rows in the order of the plan (the tensor-core tiles read them with one TMA descriptor): xg[row] = h[row_tok[row]]
template <class T>
__global__ void k_moe_gather(const T* __restrict__ h, const int32_t* __restrict__ row_tok, int W, T* __restrict__ xg) {
  pdl_launch_dependents();
  pdl_wait();
  const int row = blockIdx.x;
  const T* src = h + (size_t)row_tok[row] * W;
  T* dst = xg + (size_t)row * W;
  if ((W * (int)sizeof(T)) % 16 == 0) {
    for (int c = threadIdx.x; c < W * (int)sizeof(T) / 16; c += blockDim.x) reinterpret_cast<uint4*>(dst)[c] = reinterpret_cast<const uint4*>(src)[c];
  } else {
    for (int c = threadIdx.x; c < W; c += blockDim.x) dst[c] = src[c];
  }
}

}  // namespace dn
