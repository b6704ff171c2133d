// dn_rows.cuh -- the decoder layer's products for chunks of 1 .. ROWS_MAX tokens: every weight is read once and meets all the tokens on
// the tensor cores (dn_rows_mma.cuh).  Bound by the weights' bytes.  Three tokens behind 256, Llama-8B sizes: 253 us a layer as chunks of
// 2 + 1 on the row kernels (two passes), 106 as one; gate and up 37.1 us, 6.3 TB/s.  From 17 tokens on the GEMM takes over (calls timed with
// their copies, before the launches were programmatic: Llama-8B sizes 16 tokens 155 us here, 17 there 179; Qwen-32B sizes 268 / 257).
// A block takes 16 features (gate / up: the same 16 of both matrices).  The first weights are asked for before the kernel in front has
// ended (programmatic dependent launch); what that kernel wrote is read after the wait.  Rounding as in the GEMM's epilogues (dn_gemm_tc.cuh).
#pragma once
#include "dn_gemm_tc.cuh"
#include "dn_rows_mma.cuh"

namespace dn {

constexpr int ROWS_MAX = 16;
struct RowsParams {
  TcSeg seg[TC_SEGS];      // features of each product, as the GEMM takes them
  const bf16* w[TC_SEGS];  // their weights; EPI_SWIGLU: w[0] gate, w[1] up
  int nseg, T, K;
  const bf16* x;           // [T][K]
  const bf16* resid; int ldr;
  // one token's experts (MOE): product i is that of expert sel[i] with the matrices table[m0 + sel], EPI_SWIGLU also table[m1 + sel]; its
  // result goes to seg[0].Y + i * seg[0].ldy, its row is x + i * ldx
  const bf16* const* table; const int32_t* sel; int m0, m1, ldx;
};

template <int EPI, int NT, int U, bool MOE = false>
__global__ void __launch_bounds__(RM_THREADS, EPI == EPI_SWIGLU || U == 8 ? 2 : 3) k_rows(const __grid_constant__ RowsParams p) {
  constexpr int TILES = EPI == EPI_SWIGLU ? 2 : 1;
  __shared__ float red[RM_WARPS * TILES * NT * 128];
  pdl_launch_dependents();
  int blk = blockIdx.x, si = 0;
  const bf16* x = p.x;
  if (MOE) {
    const int nb = (p.seg[0].N + 15) / 16;
    si = blk / nb;
    blk -= si * nb;
    x += (size_t)si * p.ldx;
  } else if (EPI == EPI_STORE)
    for (; si + 1 < p.nseg; ++si) {
      const int nb = (p.seg[si].N + 15) / 16;
      if (blk < nb) break;
      blk -= nb;
    }
  const TcSeg& sg = p.seg[MOE ? 0 : si];
  const bf16* w[TILES];
  int r0[TILES];
#pragma unroll
  for (int i = 0; i < TILES; ++i) { w[i] = MOE ? nullptr : p.w[si + i]; r0[i] = blk * 16; }
  if (MOE) {      // which matrices is known only behind the wait
    pdl_wait();
    const int e = p.sel[si];
#pragma unroll
    for (int i = 0; i < TILES; ++i) w[i] = p.table[(i ? p.m1 : p.m0) + e];
    rows_mma_block<TILES, NT, U>(w, r0, sg.N, x, p.T, p.K, red);
  } else rows_mma_block<TILES, NT, U>(w, r0, sg.N, x, p.T, p.K, red, [] { pdl_wait(); });
  const int q = threadIdx.x >> 7, at = threadIdx.x & 127, row = at & 15, t = 8 * q + (at >> 4), n = blk * 16 + row;      // neighbouring threads: neighbouring features
  if (q >= NT || t >= p.T || n >= sg.N) return;
  const int slot = row * 8 + (at >> 4);
  const float a = rows_mma_sum<TILES, NT>(red, 0, slot, q);
  float y;
  if (EPI == EPI_STORE) y = a + (sg.bias ? __bfloat162float(sg.bias[n]) : 0.f);
  else if (EPI == EPI_RESID) y = __fadd_rn(__bfloat162float(p.resid[(size_t)t * p.ldr + n]), bf16r(a));
  else {
    const float g = bf16r(a), u = bf16r(rows_mma_sum<TILES, NT>(red, TILES - 1, slot, q));
    const float sg1 = bf16r(1.0f / (1.0f + expf(-g)));
    y = __fmul_rn(bf16r(__fmul_rn(g, sg1)), u);
  }
  sg.Y[(size_t)(MOE ? si : t) * sg.ldy + n] = __float2bfloat16_rn(y);
}

}  // namespace dn
