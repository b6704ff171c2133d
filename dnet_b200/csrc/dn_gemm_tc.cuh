// dn_gemm_tc.cuh -- GEMMs of prompt portions on the 5th-gen tensor cores (tcgen05 + TMEM), operands staged by TMA
// (cp.async.bulk.tensor.2d, SWIZZLE_128B), two CTAs on one tile (cta_group::2), warp-specialised: warp 0 = TMA producer,
// warp 1 = MMA issuer (one thread of the leading CTA), warp 2 = TMEM allocator, warps 4-11 = epilogue (tcgen05.ld).
//
//   Y[T, N] = X[T, K] . W[N, K]^T        bf16 operands, fp32 accumulate in TMEM
//
// "swap-AB" orientation: the WEIGHT tile is the MMA's A operand (M = 256 rows per pair of CTAs, 128 each, one TMEM lane a row) and
// the TOKEN tile is B (up to 256 tokens = TMEM columns, half of them staged by each CTA), because prefill chunks have few tokens
// and many output features; both operands are K-major in shared memory, exactly what TMA produces from row-major [rows, K] tensors.
// A stage is three copies of a CTA: 64 + 64 rows of weights, and its half of the tokens in one box.  (With the tokens in boxes of 32 rows the issue of a stage's
// copies, by one thread, took longer than its MMAs: 18,944 features of 4,096, 2,048 tokens 314 us -> 212; 1,000 tokens 174 -> 120.)
// An SM takes about 64 bytes a cycle from L2: a 128 x 128 tile of one CTA needs 128 for full tensor rate, 128 x 256 of a pair's
// half 64.  A tile is therefore as wide in tokens as the chunk allows (TcPlan), and where that leaves too few tiles for the SMs
// the reduction is split over the S pairs of a cluster, which add their accumulators through distributed shared memory in a fixed
// order.  With few tokens one CTA may take a tile of half as many features (CG = 1, tc_plan).  Whole rounds of tiles are walked persistently with two accumulator sets in TMEM; the tiles of a last, mostly empty round
// are cut into narrower pieces.
//
// Up to TC_SEGS products that read the same X run in one launch (q, k, v): tiles of all of them fill the SMs together.
//
// Epilogues (fused, same rounding points as the decode kernels / oracle):
//   EPI_STORE  : y = T(acc + bias)                        -> Y[t][n]
//   EPI_RESID  : y = T(resid[t][n] + T(acc))              -> Y[t][n]
//   EPI_SWIGLU : gate and up rows share the token tile; g = T(acc_g), u = T(acc_u),
//                s = T(sigmoid g), a = T(g s), m = T(a u)  -> Y[t][n]
//   EPI_STORE_F32 : the fp32 accumulator itself (+ bias)      -> ((float*)Y)[t][n]   (outputs that join an fp32
//                residual or feed fp32 gates)
//   EPI_GEGLU  : two weights like EPI_SWIGLU; y = T(gelu_tanh(acc_g) * acc_u), the activation and the product
//                in fp32 with one rounding                     -> Y[t][n]
//   EPI_TANH   : y = T(tanh(acc))                              -> Y[t][n]
//   EPI_CGLU   : two weights; g = min(acc_g, limit), u = clamp(acc_u, -limit, limit), y = T(g sigmoid(1.702 g) (u + 1))
//   EPI_SGLU   : two weights; y = T(silu(acc_g) * acc_u), in fp32 with one rounding
//   EPI_RELU2  : y = T(relu(acc + bias)^2)
//   EPI_GELU_TAB : y = T(gelu_tanh(acc) * tab[row[t] tab_ld + n]), in fp32 with one rounding
//   EPI_JOIN   : an fp32 residual takes the product in, x[t][n] += acc mul ls[n], and the norm that follows is elementwise:
//                nh[t][n] = T(tanh(alpha x) w + b), or T(x) without an alpha (ls, nh optional; no Y)
// Two-weight forms stage 64 gate and 64 up rows a CTA.
//
// GROUPED: one launch over many weight matrices of one shape (routed experts).  The token rows are sorted by matrix
// into tiles that never span two matrices; a device table gives every token tile its matrix, first row
// and row count, and the weights' TMA descriptors lie in an array in global memory (written by the host before the
// launch).  The number of token tiles is read from device memory, so the host never learns the routing.
#pragma once
#include <cuda.h>
#include <math.h>
#include <string.h>
#include "dn_megakernel.cuh"

namespace dn {

enum { EPI_STORE = 0, EPI_RESID = 1, EPI_SWIGLU = 2, EPI_STORE_F32 = 3, EPI_GEGLU = 4, EPI_CGLU = 5, EPI_TANH = 6, EPI_SGLU = 7, EPI_RELU2 = 8, EPI_GELU_TAB = 9, EPI_JOIN = 10 };
__host__ __device__ constexpr bool epi_two_weights(int epi) { return epi == EPI_SWIGLU || epi == EPI_GEGLU || epi == EPI_CGLU || epi == EPI_SGLU; }

constexpr int TC_BK = 64;         // k-step: 64 bf16 = 128 bytes = one swizzle span
constexpr int TC_WBOX = 64;       // rows of a weight descriptor's box
constexpr int TC_XBOX = 32;       // rows of an activation descriptor's box, or twice, three or four times as many (TcMaps::x)
constexpr int TC_XMAPS = 4;
constexpr int TC_WMAX = 256;      // tokens of a tile at most
constexpr int TC_THREADS = 384;
constexpr int TC_EWARPS = 8;
constexpr int TC_SEGS = 4;
constexpr int TC_A_BYTES = 128 * TC_BK * 2;                       // a CTA's weight rows of a stage
constexpr int TC_RING = 6 * (TC_A_BYTES + 128 * TC_BK * 2);       // bytes of all stages; also holds a split tile's partial sums
constexpr int TC_MAX_STAGES = 10;
constexpr int TC_PITCH = 36, TC_BOX = 16 * TC_PITCH;              // an epilogue warp's [16 tokens][32 features] in floats (16-byte rows, no bank conflicts)
constexpr int TC_XCH = TC_EWARPS * TC_BOX * 4;
constexpr int TC_SMEM = TC_RING + TC_XCH + 1024 + 512;

struct TcSeg {                    // one product of a launch
  int N, ldy;                     // output features, leading dimension of Y (elements)
  bf16* Y;
  const bf16* bias;               // [N] or null
  int vec;                        // rows of Y (and of what the epilogue reads) start on 16-byte boundaries (set by tc_launch)
};
struct TcMaps {
  CUtensorMap w[TC_SEGS];         // two-weight forms: [0] gate, [1] up
  CUtensorMap x[TC_XMAPS];        // the tokens, in boxes of TC_XBOX (i + 1) rows
};
struct TcParams {
  int T, K;                       // tokens, reduction
  int nseg;
  TcSeg seg[TC_SEGS];
  const bf16* resid;              // [T][ldr]
  int ldr;
  unsigned int* err;
  float limit;                    // EPI_CGLU
  const bf16* tab; const int32_t* row; int tab_ld;       // EPI_GELU_TAB
  float* x; const bf16* ls; float mul; const bf16 *nw, *nb, *nalpha; bf16* nh;      // EPI_JOIN, leading dimension seg[0].ldy
  // GROUPED: token tile tt uses the matrix g_tile_e[tt] on the rows [g_tile_r0[tt], + g_tile_rows[tt]) of X and Y
  const int32_t *g_tile_e, *g_tile_r0, *g_tile_rows, *g_ntiles;
  const CUtensorMap *g_mapW, *g_mapW2;      // [matrices], 64-byte aligned, in global memory
  // the plan (tc_plan)
  int width, split, stages;       // tokens of a tile, pairs that share a tile's reduction, stages of the ring
  int early;                      // launched programmatically: the first weights are asked for ahead of the tokens
};

__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
// address of this CTA's shared object in the cluster's CTA `rank`
__device__ __forceinline__ uint32_t dsmem_addr(const void* p, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void dsmem_st(uint32_t addr, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }
// all threads of all CTAs of the cluster
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) { asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory"); }
// bounded wait as mbar_wait, for a barrier that threads of other CTAs arrive on
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ void mbar_wait_cluster(uint64_t* bar, uint32_t parity, unsigned int* err) {
  if (mbar_try_wait_cluster(bar, parity)) return;
  const unsigned long long t0 = gtimer();
  for (unsigned it = 1; !mbar_try_wait_cluster(bar, parity); ++it)
    if ((it & 1023u) == 0 && gtimer() - t0 > MK_TIMEOUT_NS) { atomicExch(err, 2u); return; }
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
               : "memory");
}
// into this CTA's shared memory, counted on a barrier of the pair's leading CTA (`bar`: its cluster address)
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(smem_u32(dst)), "l"(map), "r"(bar), "r"(c0), "r"(c1)
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// arrives on the barrier at this offset in every CTA of `mask` once the pair's MMAs so far have retired
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar, uint16_t mask) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"(mask) : "memory");
}
// D[tmem] (+)= A[smem] . B[smem]^T   (kind::f16: bf16 x bf16 -> fp32)
__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// the same on both CTAs of a pair: A rows 0-127 (128-255) and the first (second) half of B's rows from the leading (other) CTA
__device__ __forceinline__ void tc_mma_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] . B[smem]^T   (A: bf16 pairs, one row a lane)
__device__ __forceinline__ void tc_mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// K-major, SWIZZLE_128B shared-memory matrix descriptor (cute::UMMA::SmemDescriptor layout):
//  [0,14) start address >> 4 | [16,30) leading byte offset >> 4 (unused for swizzled K-major) |
//  [32,46) stride byte offset >> 4 = 1024 B between 8-row groups | [46,48) version = 1 (sm_100) |
//  [61,64) layout type = 2 (SWIZZLE_128B)
__device__ __forceinline__ uint64_t tc_smem_desc(const void* smem_ptr) {
  const uint32_t addr = smem_u32(smem_ptr);
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFF) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// instruction descriptor (cute::UMMA::InstrDescriptor): c_format F32 (1) at [4,6), a/b format BF16 (1)
// at [7,10)/[10,13), a/b K-major (0) at 15/16, N>>3 at [17,23), M>>4 at [24,29)
__device__ __forceinline__ uint32_t tc_instr_desc(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
// MN-major, SWIZZLE_128B operand: 64 contiguous elements along N per 128-byte row, 8 k-rows per
// 1024-byte atom; LBO = bytes between N atoms (dims 0-63 -> 64-127), SBO = bytes between k groups
__device__ __forceinline__ uint64_t tc_smem_desc_mn(const void* smem_ptr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  const uint32_t addr = smem_u32(smem_ptr);
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFF) >> 4);
  d |= (uint64_t)(lbo_bytes >> 4) << 16;
  d |= (uint64_t)(sbo_bytes >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// byte offset of the 16-byte chunk (row r, chunk c of 16) inside a [2 halves][128 rows][128 B] swizzled tile
__device__ __forceinline__ uint32_t at_swz(int r, int c) {
  return (uint32_t)((c >> 3) * 16384 + r * 128 + (((c & 7) ^ (r & 7)) << 4));
}

// 32 lanes x 16 consecutive fp32 columns of this warp's TMEM quarter
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
// 32 consecutive 32-bit columns of this warp's TMEM quarter; the registers are valid after tm_wait_ld and tm_pin
__device__ __forceinline__ void tm_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
        "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
        "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tm_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// no use of r moves above this point
__device__ __forceinline__ void tm_pin(uint32_t (&r)[32]) {
#pragma unroll
  for (int i = 0; i < 32; i += 8)
    asm volatile("" : "+r"(r[i]), "+r"(r[i + 1]), "+r"(r[i + 2]), "+r"(r[i + 3]), "+r"(r[i + 4]), "+r"(r[i + 5]), "+r"(r[i + 6]), "+r"(r[i + 7]));
}
__device__ __forceinline__ void tm_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// exponential of the special-function unit (a few units in the last place of fp32, far inside what the bf16 operands carry)
__device__ __forceinline__ float tc_ex2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }

// a launch's tiles.  Rounds of whole tiles, then the last tiles cut `cut` times along the tokens, so that their round is shorter
struct TcTiles {
  int t_tiles, whole, cut, units;
};
__host__ __device__ __forceinline__ TcTiles tc_tiles(int n_tiles, int t_tiles, int width, int split, int pairs) {
  TcTiles r;
  r.t_tiles = t_tiles;
  const int total = n_tiles * t_tiles, rest = total % pairs;
  r.cut = split > 1 || rest == 0 ? 1 : rest * 4 <= pairs && width % 128 == 0 ? 4 : rest * 2 <= pairs && width % 64 == 0 ? 2 : 1;
  r.whole = r.cut > 1 ? total - rest : total;
  r.units = r.whole + (total - r.whole) * r.cut;
  return r;
}
// bytes of a stage of tiles of w tokens: a CTA's weight rows and its share of the tokens in whole boxes
__host__ __device__ constexpr int tc_stage_bytes(int w, int cg) { return TC_A_BYTES + (w / cg + TC_XBOX - 1) / TC_XBOX * (TC_XBOX * TC_BK * 2); }
template <int EPI>
__host__ __device__ constexpr int tc_tile_rows(int cg = 2) { return (epi_two_weights(EPI) ? 64 : 128) * cg; }      // output features of a tile

// CG: CTAs that work on one tile (a pair, or one with half of a pair's rows)
template <int EPI, bool GROUPED = false, int CG = 2>
__global__ void __launch_bounds__(TC_THREADS, 1) k_gemm_tc(const __grid_constant__ TcMaps maps, const __grid_constant__ TcParams p) {
  constexpr bool GLU = epi_two_weights(EPI);
  constexpr int ROWS = tc_tile_rows<EPI>(CG);
  pdl_launch_dependents();
  if (GROUPED) pdl_wait();        // the tiles are a table that the kernel in front has written
  extern __shared__ __align__(1024) unsigned char tc_smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~(uintptr_t)1023);
  float* xch = reinterpret_cast<float*>(smem + TC_RING);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + TC_RING + TC_XCH);      // counted in the leading CTA
  uint64_t* empty = full + TC_MAX_STAGES;
  uint64_t* tmem_full = empty + TC_MAX_STAGES;   // [2]
  uint64_t* tmem_empty = tmem_full + 2;          // [2], counted in the leading CTA
  uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t crank = cluster_rank(), lead = crank / CG * CG;
  const int rank = (int)(crank % CG), part = (int)(crank / CG);      // place in the pair; which share of a split reduction
  const int S = p.split, W = p.width, stages = p.stages;
  int n_tiles = 0;
  for (int i = 0; i < p.nseg; ++i) n_tiles += (p.seg[i].N + ROWS - 1) / ROWS;
  const int pairs = (int)gridDim.x / (CG * S), pair = (int)blockIdx.x / (CG * S);      // (a cluster counts once)
  const TcTiles tl = tc_tiles(n_tiles, GROUPED ? *p.g_ntiles : (p.T + W - 1) / W, W, S, pairs);
  const int k_all = p.K / TC_BK, k0 = (int)((long long)k_all * part / S), k1 = (int)((long long)k_all * (part + 1) / S);
  const int stage_bytes = tc_stage_bytes(W, CG);

  if (threadIdx.x == 0) {
    for (int i = 0; i < stages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&tmem_full[i], 1); mbar_init(&tmem_empty[i], CG * TC_EWARPS); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {                // TMEM allocation (a warp of each CTA of the pair), address lands in shared memory
    if (CG == 2) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_base_slot)) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_base_slot)) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_base_slot;

  // a unit's tile: segment and first row of the weights, first token and how many
  struct Tile { int seg, n0, e, t0, t_end, cols; };
  auto tile_of = [&](int u) {
    Tile r;
    int tile = u, sub = 0;
    if (u >= tl.whole) { tile = tl.whole + (u - tl.whole) / tl.cut; sub = (u - tl.whole) % tl.cut; }
    const int w = u >= tl.whole ? W / tl.cut : W;
    const int tt = tile % tl.t_tiles;             // token tiles of one weight tile run back to back (weights hit L2)
    int nt = tile / tl.t_tiles;
    r.seg = 0;
    while (r.seg + 1 < p.nseg && nt >= (p.seg[r.seg].N + ROWS - 1) / ROWS) { nt -= (p.seg[r.seg].N + ROWS - 1) / ROWS; ++r.seg; }
    r.n0 = nt * ROWS;
    r.e = 0;
    if (GROUPED) {
      r.e = p.g_tile_e[tt];
      r.t0 = p.g_tile_r0[tt] + sub * w;
      r.t_end = min(r.t0 + w, p.g_tile_r0[tt] + p.g_tile_rows[tt]);
    } else {
      r.t0 = tt * W + sub * w;
      r.t_end = min(r.t0 + w, p.T);
    }
    r.cols = S > 1 ? W : min(w, (max(r.t_end - r.t0, 1) + 15) & ~15);      // a pair computes whole sixteens of tokens
    return r;
  };

  // The producer asks for the weights of a ring's worth of stages before the kernel in front has ended (programmatic dependent launch); what that one
  // wrote -- tokens, residuals -- is read behind the wait.  45 tokens, Llama-8B sizes, a layer: 157 us without, 148.  An ordinary launch has nothing to wait
  // for, and there the first stage's tokens would come behind the weights of all others.
  if (warp != 0 && !GROUPED) pdl_wait();
  if (warp == 0) {
    // ===================== TMA producer (each CTA its own rows; bytes counted by the leading CTA) =====================
    if (lane == 0) {
      int stage = 0; uint32_t phase = 0;
      int early = 0;              // k-steps of the first tile whose weights are on their way
      for (int u = pair; u < tl.units; u += pairs) {
        const Tile tl_ = tile_of(u);
        const CUtensorMap *mw = &maps.w[tl_.seg], *mw2 = &maps.w[GLU ? 1 : tl_.seg];
        if (GROUPED) {      // descriptors read from global memory: make the host's writes visible to the TMA unit
          mw = p.g_mapW + tl_.e;
          mw2 = GLU ? p.g_mapW2 + tl_.e : mw;
          asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(mw) : "memory");
          if (GLU) asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(mw2) : "memory");
        }
        const int r0 = GLU ? tl_.n0 + rank * 64 : tl_.n0 + rank * 128, r1 = GLU ? r0 : r0 + 64;
        const int x0 = tl_.t0 + rank * (tl_.cols / CG), boxes = (tl_.cols / CG + TC_XBOX - 1) / TC_XBOX;
        const CUtensorMap* mx = &maps.x[boxes - 1];
        const uint32_t bytes = (uint32_t)CG * (TC_A_BYTES + boxes * (TC_XBOX * TC_BK * 2));
        auto weights = [&](int st, int ks) {
          const uint32_t bar = dsmem_addr(&full[st], lead);
          if (rank == 0) mbar_arrive_expect_tx(&full[st], bytes);
          unsigned char* sa = smem + (size_t)st * stage_bytes;
          if (CG == 2) {
            tma_load_2d_pair(sa, mw, ks * TC_BK, r0, bar);
            tma_load_2d_pair(sa + TC_A_BYTES / 2, mw2, ks * TC_BK, r1, bar);
          } else {
            tma_load_2d(sa, mw, ks * TC_BK, r0, &full[st]);
            tma_load_2d(sa + TC_A_BYTES / 2, mw2, ks * TC_BK, r1, &full[st]);
          }
        };
        if (!GROUPED && u == pair) {
          if (p.early) early = min(stages, k1 - k0);
          for (int i = 0; i < early; ++i) weights(i, k0 + i);
          pdl_wait();
        }
        for (int ks = k0; ks < k1; ++ks) {
          if (early > 0) --early;
          else {
            mbar_wait(&empty[stage], phase ^ 1u, p.err);
            weights(stage, ks);
          }
          unsigned char* sx = smem + (size_t)stage * stage_bytes + TC_A_BYTES;
          if (CG == 2) tma_load_2d_pair(sx, mx, ks * TC_BK, x0, dsmem_addr(&full[stage], lead));
          else tma_load_2d(sx, mx, ks * TC_BK, x0, &full[stage]);
          if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ===================== MMA issuer (one thread of the leading CTA) =====================
    if (lane == 0 && rank == 0) {
      const uint16_t both = (uint16_t)(3u << lead);
      int stage = 0; uint32_t phase = 0;
      uint32_t it = 0;
      for (int u = pair; u < tl.units; u += pairs, ++it) {
        const uint32_t idesc = tc_instr_desc(128 * CG, tile_of(u).cols);
        const uint32_t ab = it & 1u, acc_phase = (it >> 1) & 1u, tacc = tmem_base + ab * TC_WMAX;
        mbar_wait_cluster(&tmem_empty[ab], acc_phase ^ 1u, p.err);    // both CTAs' epilogues drained this accumulator set
        tc_fence_after();
        for (int ks = k0; ks < k1; ++ks) {
          mbar_wait(&full[stage], phase, p.err);      // (bytes of both CTAs' copies; arrived on by this CTA alone)
          tc_fence_after();
          unsigned char* sa = smem + (size_t)stage * stage_bytes;
          const uint64_t adesc = tc_smem_desc(sa), bdesc = tc_smem_desc(sa + TC_A_BYTES);
#pragma unroll
          for (int k = 0; k < TC_BK / 16; ++k) {      // +32 bytes (>>4 = 2) per UMMA_K inside the swizzle span
            if (CG == 2) tc_mma_pair(tacc, adesc + (uint64_t)(2 * k), bdesc + (uint64_t)(2 * k), idesc, (ks > k0 || k) ? 1u : 0u);
            else tc_mma(tacc, adesc + (uint64_t)(2 * k), bdesc + (uint64_t)(2 * k), idesc, (ks > k0 || k) ? 1u : 0u);
          }
          if (CG == 2) tc_commit_pair(&empty[stage], both);        // both CTAs' stages are reusable once these MMAs retire
          else tc_commit(&empty[stage]);
          if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
        if (CG == 2) tc_commit_pair(&tmem_full[ab], both);         // accumulator complete -> both epilogues
        else tc_commit(&tmem_full[ab]);
      }
    }
  }

  // ===================== epilogue: TMEM -> registers -> shared memory -> global =====================
  const int qd = warp & 3, half = (warp - 4) >> 2;    // TMEM lanes [32 qd, 32 qd + 32); half of the columns
  const uint32_t lane_off = (uint32_t)(qd * 32) << 16;
  // Columns [c_lo, c_hi) of the accumulator at tacc, sixteen at a time.  A TMEM lane is a feature and a column a token; global memory wants the
  // features of a token side by side, so every chunk turns in shared memory (`box`, [16 tokens][32 features] a warp) and a thread finishes
  // eight features of a token: 16-byte loads and stores, 64 bytes a token and warp.  (Straight from the lanes every store is 2 bytes a thread:
  // the epilogue of a 256 x 256 tile then took longer than its 64 k-steps.)
  // With parts: `got` holds the other parts' sums [S][per][128], added in the order of the parts, whichever of them adds.
  float* box = xch + (warp - 4) * TC_BOX;
  const int tq = lane >> 2, fq = (lane & 3) * 8, up = qd >> 1;
  constexpr int PASSES = GLU ? 1 : 2;       // of eight tokens
  auto emit = [&](const Tile& tl_, uint32_t tacc, int c_lo, int c_hi, const float* got, int per) {
    const TcSeg& sg = p.seg[tl_.seg];
    const int n = GLU ? tl_.n0 + rank * 64 + (qd & 1) * 32 + fq : tl_.n0 + rank * 128 + qd * 32 + fq;      // first of the thread's eight features
    const int n_have = min(8, sg.N - n);
    const bool vec = n_have == 8 && sg.vec;
    float bias[8], jls[8], jw[8], jb[8], ja = 0.f;
    if (EPI == EPI_STORE || EPI == EPI_STORE_F32 || EPI == EPI_RELU2)
#pragma unroll
      for (int i = 0; i < 8; ++i) bias[i] = sg.bias != nullptr && i < n_have ? __bfloat162float(sg.bias[n + i]) : 0.f;
    if (EPI == EPI_JOIN) {
      if (p.nalpha) ja = 2.885390081777927f * __bfloat162float(*p.nalpha);      // 2 log2(e) alpha
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        jls[i] = p.ls && i < n_have ? p.mul * __bfloat162float(p.ls[n + i]) : p.mul;
        jw[i] = p.nalpha && i < n_have ? __bfloat162float(p.nw[n + i]) : 0.f;
        jb[i] = p.nalpha && i < n_have ? __bfloat162float(p.nb[n + i]) : 0.f;
      }
    }
    // what a joining epilogue reads is asked for a chunk ahead
    constexpr bool OPS = EPI == EPI_JOIN || EPI == EPI_GELU_TAB || EPI == EPI_RESID;
    float nxt[OPS ? 2 : 1][8], op[OPS ? 2 : 1][8];
    auto ahead = [&](int c) {
#pragma unroll
      for (int z = 0; z < 2; ++z) {
        const int cc = c + z * 8 + tq, t = tl_.t0 + cc;
        if (t >= tl_.t_end || cc >= c_hi || n_have <= 0) continue;
        float* d = nxt[OPS ? z : 0];
        if (EPI == EPI_JOIN) {
          const float* src = p.x + (size_t)t * sg.ldy + n;
          if (vec) {
            *reinterpret_cast<float4*>(d) = *reinterpret_cast<const float4*>(src);
            *reinterpret_cast<float4*>(d + 4) = *reinterpret_cast<const float4*>(src + 4);
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) if (i < n_have) d[i] = src[i];
          }
        } else {
          const bf16* src = EPI == EPI_RESID ? p.resid + (size_t)t * p.ldr + n : p.tab + (size_t)p.row[t] * p.tab_ld + n;
          if (vec) {
            const uint4 v = *reinterpret_cast<const uint4*>(src);
            d[0] = bf_lo(v.x); d[1] = bf_hi(v.x); d[2] = bf_lo(v.y); d[3] = bf_hi(v.y); d[4] = bf_lo(v.z); d[5] = bf_hi(v.z); d[6] = bf_lo(v.w); d[7] = bf_hi(v.w);
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) if (i < n_have) d[i] = __bfloat162float(src[i]);
          }
        }
      }
    };
    if (OPS) ahead(c_lo);
#pragma unroll 1
    for (int c = c_lo; c < c_hi; c += 16) {
      float v[16];
      tc_ld16(tacc + lane_off + c, v);
      if (S > 1) {
        float s[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) s[j] = 0.f;
        for (int q = 0; q < S; ++q)
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (c + j < c_hi) s[j] += q == part ? v[j] : got[((size_t)q * per + (c + j - part * per)) * 128 + qd * 32 + lane];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = s[j];
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) box[j * TC_PITCH + lane] = v[j];
      if (OPS) {
#pragma unroll
        for (int z = 0; z < 2; ++z)
#pragma unroll
          for (int i = 0; i < 8; ++i) op[OPS ? z : 0][i] = nxt[OPS ? z : 0][i];
        if (c + 16 < c_hi) ahead(c + 16);
      }
      // (two weights: lanes 0-63 hold the gate products and 64-127 the up products of the same features; each of the two warps finishes
      // eight of the sixteen tokens)
      if (GLU) asm volatile("bar.sync %0, 64;" ::"r"(2 + half * 2 + (qd & 1)) : "memory");
      else __syncwarp();
      const float* box_g = GLU ? xch + (warp - 4 - 2 * up) * TC_BOX : box;
      const float* box_u = GLU ? box_g + 2 * TC_BOX : box;
#pragma unroll
      for (int z = 0; z < PASSES; ++z) {
        const int j = (GLU ? up : z) * 8 + tq, t = tl_.t0 + c + j;
        if (t >= tl_.t_end || c + j >= c_hi || n_have <= 0) continue;
        float a[8], b[8], y[8];
        *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(box_g + j * TC_PITCH + fq);
        *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(box_g + j * TC_PITCH + fq + 4);
        if (GLU) {
          *reinterpret_cast<float4*>(b) = *reinterpret_cast<const float4*>(box_u + j * TC_PITCH + fq);
          *reinterpret_cast<float4*>(b + 4) = *reinterpret_cast<const float4*>(box_u + j * TC_PITCH + fq + 4);
        }
        const float* o = op[OPS ? z : 0];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (EPI == EPI_STORE || EPI == EPI_STORE_F32) {
            y[i] = a[i] + bias[i];
          } else if (EPI == EPI_JOIN) {
            y[i] = o[i] + a[i] * jls[i];
          } else if (EPI == EPI_GELU_TAB) {
            y[i] = 0.5f * a[i] * (1.0f + tanhf(0.7978845608028654f * (a[i] + 0.044715f * a[i] * a[i] * a[i]))) * o[i];
          } else if (EPI == EPI_GEGLU) {
            y[i] = 0.5f * a[i] * (1.0f + tanhf(0.7978845608028654f * (a[i] + 0.044715f * a[i] * a[i] * a[i]))) * b[i];
          } else if (EPI == EPI_TANH) {
            y[i] = tanhf(a[i]);
          } else if (EPI == EPI_SGLU) {
            y[i] = a[i] / (1.0f + expf(-a[i])) * b[i];
          } else if (EPI == EPI_RELU2) {
            const float r = fmaxf(a[i] + bias[i], 0.f);
            y[i] = r * r;
          } else if (EPI == EPI_CGLU) {
            const float g = fminf(a[i], p.limit), u = fminf(fmaxf(b[i], -p.limit), p.limit);
            y[i] = g / (1.0f + expf(-1.702f * g)) * (u + 1.0f);
          } else if (EPI == EPI_RESID) {
            y[i] = __fadd_rn(o[i], bf16r(a[i]));
          } else {
            const float g = bf16r(a[i]), u = bf16r(b[i]);
            const float s = bf16r(1.0f / (1.0f + expf(-g)));
            y[i] = __fmul_rn(bf16r(__fmul_rn(g, s)), u);
          }
        }
        if (EPI == EPI_STORE_F32 || EPI == EPI_JOIN) {
          float* dst = (EPI == EPI_JOIN ? p.x : reinterpret_cast<float*>(sg.Y)) + (size_t)t * sg.ldy + n;
          if (vec) {
            *reinterpret_cast<float4*>(dst) = *reinterpret_cast<const float4*>(y);
            *reinterpret_cast<float4*>(dst + 4) = *reinterpret_cast<const float4*>(y + 4);
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) if (i < n_have) dst[i] = y[i];
          }
          if (EPI == EPI_STORE_F32 || !p.nh) continue;
        }
        if (EPI == EPI_JOIN) {      // the norm that follows.  tanh(z) = 1 - 2 / (1 + e^2z): an absolute error of a few 1e-7, far below the rounding of the result
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (p.nalpha) y[i] = fmaf(1.f - __fdividef(2.f, 1.f + exp2f(fminf(ja * y[i], 80.f))), jw[i], jb[i]);
        }
        bf16* dst = (EPI == EPI_JOIN ? p.nh : sg.Y) + (size_t)t * sg.ldy + n;
        if (vec) {
          __align__(16) bf16 w[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) w[i] = __float2bfloat16_rn(y[i]);
          *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(w);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) if (i < n_have) dst[i] = __float2bfloat16_rn(y[i]);
        }
      }
      // the box may be written again
      if (GLU) asm volatile("bar.sync %0, 64;" ::"r"(2 + half * 2 + (qd & 1)) : "memory");
      else __syncwarp();
    }
  };

  if (S == 1) {
    if (warp >= 4) {
      uint32_t it = 0;
      for (int u = pair; u < tl.units; u += pairs, ++it) {
        const Tile tl_ = tile_of(u);
        const uint32_t ab = it & 1u, acc_phase = (it >> 1) & 1u;
        const int hw = tl_.cols / 2;
        mbar_wait(&tmem_full[ab], acc_phase, p.err);
        __syncwarp();
        tc_fence_after();
        emit(tl_, tmem_base + ab * TC_WMAX, half * hw, half * hw + hw, nullptr, 0);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(dsmem_addr(&tmem_empty[ab], lead));
      }
    }
  } else {
    // one tile a cluster: the S pairs' accumulators meet, every pair finishes 1 / S of the columns
    float* got = reinterpret_cast<float*>(smem);      // [S][per][128], over the ring: no stage is in use any more
    const int per = W / S;
    const Tile tl_ = tile_of(pair);
    if (warp >= 4) {
      mbar_wait(&tmem_full[0], 0u, p.err);
      __syncwarp();
      tc_fence_after();
    }
    __syncwarp();
    cluster_sync();                   // every pair's MMAs have read their stages
    if (warp >= 4) {
      const int row = qd * 32 + lane;
      for (int q = 0; q < S; ++q) {
        if (q == part) continue;
        const uint32_t dst = dsmem_addr(got + (size_t)part * per * 128 + row, (uint32_t)(CG * q + rank));
        for (int c = half * (per / 2); c < (half + 1) * (per / 2); c += 8) {
          uint32_t r[8];
          asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                       : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                       : "r"(tmem_base + lane_off + q * per + c));
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 8; ++j) dsmem_st(dst + (uint32_t)((c + j) * 512), __uint_as_float(r[j]));
        }
      }
    }
    __syncwarp();
    cluster_sync();                   // the other pairs' sums are here
    if (warp >= 4) {
      const int lo = part * per + half * (per / 2);
      emit(tl_, tmem_base, lo, lo + per / 2, got, per);
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();                     // nobody leaves while the pair's other CTA may still read its memory or count on its barriers
  if (warp == 2) {
    tc_fence_after();
    if (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
  }
}

// ---------------------------------------------------------------------------------
// the plan of a launch (host).  Internal linkage: a process may load both libraries, and the statics of shared inline functions would be one object
// ---------------------------------------------------------------------------------
struct TcPlan { int width, split, stages, grid, cg; };      // cg: CTAs of a tile
static inline int tc_stages(int width, int cg = 2) {
  const int s = TC_RING / tc_stage_bytes(width, cg);
  return s < TC_MAX_STAGES ? s : TC_MAX_STAGES;
}
static inline void tc_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at, int grid, int cluster, cudaStream_t s) {
  memset(cfg, 0, sizeof(*cfg));
  cfg->gridDim = dim3(grid);
  cfg->blockDim = dim3(TC_THREADS);
  cfg->dynamicSmemBytes = TC_SMEM;
  cfg->stream = s;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = cluster;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  cfg->attrs = at;
  cfg->numAttrs = 1;
}
// clusters of n CTAs that run at once (asked of the device once; the SMs of a processing cluster hold whole ones: 33 of 4, 15 of 8)
static inline int tc_clusters(int n, int sms) {
  static int at_once[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  if (at_once[n] == 0) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[1];
    int c = 0;
    tc_config(&cfg, at, n * sms, n, 0);
    if (cudaFuncSetAttribute(k_gemm_tc<EPI_STORE, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&c, k_gemm_tc<EPI_STORE, false>, &cfg) != cudaSuccess || c < 1) {
      cudaGetLastError();
      c = sms / n * 3 / 4;
    }
    at_once[n] = c > 0 ? c : 1;
  }
  return at_once[n];
}
// What a plan is expected to take, in microseconds.  A k-step takes at least 0.28 (the way of a stage through the ring) and otherwise as long
// as its bytes from L2, of which all SMs together get 10.8 TB/s (a 256-token tile's MMAs take as long as its bytes); a launch that fills
// more than half of the SMs with pairs does no better than 120 of them would.  The weights come out of DRAM at 5.6 TB/s at best.  Start and
// end of a launch cost 6, 10.5 where partial sums meet, and the epilogue of the last tile, which nothing hides, grows with its tokens.
// Against every width and split of pairs and of single CTAs at 304 shapes (512 .. 27,648 features, reductions of 512 .. 27,648, 17 .. 2,048 tokens; launches
// one behind the other, programmatic or not) the plan so chosen is the fastest or within 5 % of it at nine of ten, within 10 % at 95 of 100, and 19 % off
// at worst (5,120 features of 27,648, 2,048 tokens, at the power limit; 6,144 of 4,096, 160 tokens 16).
static inline double tc_step(int active, int w, int cg) {
  if (active > 72 && active < 120 && cg == 2) active = 120;
  const double t = active * (double)tc_stage_bytes(w, cg) / 10.8e6;
  return t > 0.28 ? t : 0.28;
}
static inline double tc_cost(int n_tiles, int T, int K, int w, int S, int cg, int sms) {
  const int groups = sms / cg, t_tiles = (T + w - 1) / w, ks = K / TC_BK;
  const double dram = n_tiles * 128.0 * cg * K * 2.0 / 5.6e6 + 7.0;
  double c;
  if (S > 1) {
    const int at_once = tc_clusters(cg * S, sms), total = n_tiles * t_tiles, rounds = (total + at_once - 1) / at_once;
    c = rounds * ((ks + S - 1) / S * tc_step((total < at_once ? total : at_once) * cg * S, w, cg) + 10.5 + 0.035 * w);
  } else {
    const TcTiles tl = tc_tiles(n_tiles, t_tiles, w, 1, groups);
    c = tl.whole / groups * (ks * tc_step(sms, w, cg)) + 6.0 + 0.024 * w;
    if (tl.whole % groups) c += ks * tc_step(cg * (tl.whole % groups), w, cg);
    if (tl.cut > 1) c += ks * tc_step(cg * (tl.units - tl.whole), w / tl.cut, cg);
  }
  return c > dram ? c : dram;
}
// Up to TC_SINGLE_TO tokens one CTA may work on a tile, of half as many features: half as many k-steps of a split reduction fit into the clusters that run at
// once (4,096 features of 14,336: 16 tiles of pairs meet 15 clusters of eight, so that two pairs share each; 32 tiles of single CTAs meet 33 of four).  45 tokens:
// 41 us with pairs, 28 so; 4,096 x 4,096 17.1 / 15.2; 5,120 x 27,648 75 / 54; where a split gains nothing both take the same, and from 200 tokens
// on most shapes want the pairs' halved copies (14,336 x 2 of 4,096, 200 tokens: 58 / 80).  A candidate of single CTAs has to be 3 % cheaper than the best before it,
// of pairs or of single CTAs, to be taken (asked once, of the best of either, the margin changes two plans of those 304, for 5 % more time).  Of the 67 shapes
// that single CTAs then take, those with a split reduction gain 12 % on average; those without one (reductions of up to 1,024) lie between 10 % less and
// 8 % more behind programmatic launches, and are even behind ordinary ones.
constexpr int TC_SINGLE_TO = 256;
// n_pair, n_single: tiles of a pair and of a single CTA along the features
static inline TcPlan tc_plan(int n_pair, int n_single, int T, int K, int sms) {
  TcPlan best{0, 1, 0, 0, 2};
  double cost = 0;
  const int ks = K / TC_BK;
  for (int cg = 2; cg >= 1; --cg) {
    if (cg == 1 && T > TC_SINGLE_TO) break;
    for (int S = 1; S <= 4; ++S) {
      if (S > 1 && ks < 8 * S) break;
      for (int w = cg == 2 ? 64 : 48; w <= (cg == 2 ? TC_WMAX : 128); w += cg == 2 ? 32 : 16) {
        if ((S > 1 && w % (16 * S)) || (w > 96 && w >= T + 32)) continue;
        const double c = tc_cost(cg == 2 ? n_pair : n_single, T, K, w, S, cg, sms);
        if (!best.width || c < cost * (cg == 1 ? 0.97 : 0.999)) { cost = c; best.width = w; best.split = S; best.cg = cg; }
      }
    }
  }
  best.stages = tc_stages(best.width, best.cg);
  const int groups = sms / best.cg;
  const TcTiles tl = tc_tiles(best.cg == 2 ? n_pair : n_single, (T + best.width - 1) / best.width, best.width, best.split, groups);
  best.grid = best.split > 1 ? best.cg * best.split * tl.units : best.cg * (tl.units < groups ? tl.units : groups);
  return best;
}
// Rows of a grouped launch's tiles: P rows over E matrices, whose shares are taken to lie within a third of the average.  A matrix with one row more than
// a tile has takes a second one, which reads its weights again and fills a few columns, so the width keeps a distance from the average; a wider
// stage leaves fewer of them for the way of 2.5 us that each takes through the ring.  (Mixtral-8x7B, 500 tokens, 125 rows an expert: a layer 780 to 816 us with
// tiles of 128 rows, 661 to 676 with 192.  Both products alone, E = 8, 16 and 64, 17 to 2,048 tokens, choices even and uneven up to 1 : E, against tiles
// of 64, 128 or 256 rows by an average alone: where averages lie just below a tile's rows 2 to 22 % less, where one expert has many times another's share
// up to 8 % more, and the same or within 2 % elsewhere.)
static inline int tc_grouped_width(int E, int P, int sms) {
  int best = 64;
  double cost = 0;
  for (int w = 64; w <= TC_WMAX; w += 32) {
    double c = 0;
    for (int i = -2; i <= 2; ++i) {
      const int rows = (int)ceil(P * (1.0 + i / 6.0) / E), tiles = (rows + w - 1) / w, cols = rows < w ? (rows + 15) & ~15 : w;
      const int bytes = tc_stage_bytes(cols, 2);
      const double way = 2.5 / tc_stages(w), copies = sms * (double)bytes / 10.8e6;
      c += tiles * (way > copies ? way : copies);
    }
    if (w == 64 || c < cost * 0.999) { cost = c; best = w; }
  }
  return best;
}
template <int EPI, bool GROUPED, int CG>
static inline cudaError_t tc_launch_as(const TcMaps& maps, const TcParams& p, const TcPlan& pl, cudaStream_t s, bool pdl) {
  static bool attr = false;
  if (!attr) {
    const cudaError_t e = cudaFuncSetAttribute(k_gemm_tc<EPI, GROUPED, CG>, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM);
    if (e != cudaSuccess) return e;
    attr = true;
  }
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[2];
  tc_config(&cfg, at, pl.grid, CG * pl.split, s);
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = pdl ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, k_gemm_tc<EPI, GROUPED, CG>, maps, p);
}
template <int EPI, bool GROUPED>
static inline cudaError_t tc_launch(const TcMaps& maps, TcParams& p, const TcPlan& pl, cudaStream_t s, bool pdl = false) {
  p.width = pl.width; p.split = pl.split; p.stages = pl.stages; p.early = pdl;
  for (int i = 0; i < p.nseg; ++i) {
    TcSeg& sg = p.seg[i];
    bool v = sg.ldy % 8 == 0 && ((uintptr_t)sg.Y & 15) == 0;
    if (EPI == EPI_RESID) v = v && p.ldr % 8 == 0 && ((uintptr_t)p.resid & 15) == 0;
    if (EPI == EPI_GELU_TAB) v = v && p.tab_ld % 8 == 0 && ((uintptr_t)p.tab & 15) == 0;
    if (EPI == EPI_JOIN) v = v && (((uintptr_t)p.x | (uintptr_t)p.nh) & 15) == 0;
    sg.vec = v;
  }
  if constexpr (!GROUPED)
    if (pl.cg == 1) return tc_launch_as<EPI, GROUPED, 1>(maps, p, pl, s, pdl);
  return tc_launch_as<EPI, GROUPED, 2>(maps, p, pl, s, pdl);
}

// ---------------------------------------------------------------------------------
// prefill helpers around the GEMMs
// ---------------------------------------------------------------------------------
// RMSNorm of T rows (same arithmetic as stage_rmsnorm): one CTA per token
__global__ void __launch_bounds__(256) k_rmsnorm_rows(const bf16* __restrict__ x, const bf16* __restrict__ w, bf16* __restrict__ out,
                                                      int K, float eps) {
  __shared__ float scratch[8];
  pdl_launch_dependents();
  pdl_wait();
  const bf16* xr = x + (size_t)blockIdx.x * K;
  bf16* o = out + (size_t)blockIdx.x * K;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float ss = 0.f;
  for (int i = threadIdx.x * 8; i < K; i += 256 * 8) {
    const uint4 v = *reinterpret_cast<const uint4*>(xr + i);
    const float f[8] = {bf_lo(v.x), bf_hi(v.x), bf_lo(v.y), bf_hi(v.y), bf_lo(v.z), bf_hi(v.z), bf_lo(v.w), bf_hi(v.w)};
#pragma unroll
    for (int j = 0; j < 8; ++j) ss = fmaf(f[j], f[j], ss);
  }
  ss = warp_sum(ss);
  if (lane == 0) scratch[warp] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) tot += scratch[i];
  const float inv = 1.0f / sqrtf(tot / (float)K + eps);
  for (int i = threadIdx.x * 8; i < K; i += 256 * 8) {
    const uint4 v = *reinterpret_cast<const uint4*>(xr + i);
    const uint4 g = *reinterpret_cast<const uint4*>(w + i);
    const float f[8] = {bf_lo(v.x), bf_hi(v.x), bf_lo(v.y), bf_hi(v.y), bf_lo(v.z), bf_hi(v.z), bf_lo(v.w), bf_hi(v.w)};
    const float gw[8] = {bf_lo(g.x), bf_hi(g.x), bf_lo(g.y), bf_hi(g.y), bf_lo(g.z), bf_hi(g.z), bf_lo(g.w), bf_hi(g.w)};
    __align__(16) bf16 ob[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) ob[j] = __float2bfloat16_rn(__fmul_rn(bf16r(__fmul_rn(f[j], inv)), gw[j]));
    *reinterpret_cast<uint4*>(o + i) = *reinterpret_cast<const uint4*>(ob);
  }
}

// RoPE on q (in place in the qkv buffer -> q_out) and k, and KV append, for T tokens.
// qkv: [T][(n_heads + 2 n_kv) * 128] bf16 (Linear outputs already rounded to bf16)
// Bound by moving the rows (512 tokens of 48 heads: 12.6 MB).  A block takes ROPE_SLOTS heads of one token: the 64 angles' cosines and sines
// once, then a thread eight pairs of dims in 16-byte words.  (A thread a number, its own sine and cosine each: 15 us for 512 tokens; now 3.7.)
constexpr int ROPE_SLOTS = 16;
__global__ void __launch_bounds__(128) k_rope_append(const bf16* __restrict__ qkv, bf16* __restrict__ q_out, bf16* __restrict__ kv_pool,
                                                     const int32_t* __restrict__ block_table, const StepState* __restrict__ st,
                                                     const float* __restrict__ inv_freq, int n_heads, int n_kv) {
  __shared__ __align__(16) float cs_s[HD / 2], sn_s[HD / 2];
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.y, pos = st->pos + t, slots = n_heads + 2 * n_kv;      // slot: q heads, then k heads, then v heads
  const int slot = blockIdx.x * ROPE_SLOTS + (threadIdx.x >> 3), d = (threadIdx.x & 7) * 8;      // dims d .. d + 7 and 64 further on
  uint4 lo = make_uint4(0u, 0u, 0u, 0u), hi = lo;
  if (slot < slots) {
    const bf16* src = qkv + ((size_t)t * slots + slot) * HD + d;
    lo = *reinterpret_cast<const uint4*>(src);
    hi = *reinterpret_cast<const uint4*>(src + HD / 2);
  }
  if (threadIdx.x < HD / 2) sincosf(__fmul_rn((float)pos, inv_freq[threadIdx.x]), &sn_s[threadIdx.x], &cs_s[threadIdx.x]);
  __syncthreads();
  if (slot >= slots) return;
  if (slot < n_heads + n_kv) {
    const uint32_t l4[4] = {lo.x, lo.y, lo.z, lo.w}, h4[4] = {hi.x, hi.y, hi.z, hi.w};
    __align__(16) bf16 ol[8], oh[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float a = (i & 1) ? bf_hi(l4[i >> 1]) : bf_lo(l4[i >> 1]), b = (i & 1) ? bf_hi(h4[i >> 1]) : bf_lo(h4[i >> 1]);
      const float cs = cs_s[d + i], sn = sn_s[d + i];
      ol[i] = __float2bfloat16_rn(__fsub_rn(__fmul_rn(a, cs), __fmul_rn(b, sn)));
      oh[i] = __float2bfloat16_rn(__fadd_rn(__fmul_rn(a, sn), __fmul_rn(b, cs)));
    }
    lo = *reinterpret_cast<const uint4*>(ol);
    hi = *reinterpret_cast<const uint4*>(oh);
  }
  bf16* dst;
  if (slot < n_heads) dst = q_out + ((size_t)t * n_heads + slot) * HD;
  else {
    const int kind = slot >= n_heads + n_kv ? 1 : 0, hrow = slot - n_heads - kind * n_kv;
    dst = kv_pool + (((size_t)block_table[pos / PAGE] * 2 + kind) * n_kv + hrow) * (PAGE * HD) + (size_t)(pos % PAGE) * HD;
  }
  *reinterpret_cast<uint4*>(dst + d) = lo;
  *reinterpret_cast<uint4*>(dst + HD / 2 + d) = hi;
}

// causal prefill attention over the paged KV: CTA = (kv head, group of QT query tokens); warp w
// serves q head kvh*G + w for each of the QT tokens; K/V tiles are staged once per CTA.
template <int G, int QT>
__global__ void __launch_bounds__(G * 32) k_attn_prefill(const bf16* __restrict__ q, const bf16* __restrict__ kv_pool,
                                                        const int32_t* __restrict__ block_table, const StepState* __restrict__ st,
                                                        bf16* __restrict__ out, int n_heads, int n_kv, int T) {
  __shared__ __align__(16) bf16 Ks[PAGE * HD];
  __shared__ __align__(16) bf16 Vs[PAGE * HD];
  __shared__ float ps[G][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kvh = blockIdx.x, t0 = blockIdx.y * QT;
  const int head = kvh * G + warp;
  const int pos0 = st->pos;
  const int nq = min(QT, T - t0);
  const int kv_max = pos0 + t0 + nq;                     // keys visible to the last query of this CTA
  const float scale = 0.08838834764831845f;
  float qv[QT][4], m[QT], l[QT], o[QT][4];
#pragma unroll
  for (int i = 0; i < QT; ++i) {
    m[i] = -INFINITY; l[i] = 0.f;
    o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
    qv[i][0] = qv[i][1] = qv[i][2] = qv[i][3] = 0.f;
    if (i < nq) {
      const uint2 u = *reinterpret_cast<const uint2*>(q + (size_t)(t0 + i) * n_heads * HD + head * HD + lane * 4);
      qv[i][0] = __fmul_rn(bf_lo(u.x), scale); qv[i][1] = __fmul_rn(bf_hi(u.x), scale);
      qv[i][2] = __fmul_rn(bf_lo(u.y), scale); qv[i][3] = __fmul_rn(bf_hi(u.y), scale);
    }
  }
  const int npages = (kv_max + PAGE - 1) / PAGE;
  for (int pg = 0; pg < npages; ++pg) {
    const int phys = block_table[pg];
    const uint4* ksrc = reinterpret_cast<const uint4*>(kv_pool + (((size_t)phys * 2 + 0) * n_kv + kvh) * (PAGE * HD));
    const uint4* vsrc = reinterpret_cast<const uint4*>(kv_pool + (((size_t)phys * 2 + 1) * n_kv + kvh) * (PAGE * HD));
    const int ntok = min(PAGE, kv_max - pg * PAGE);
    for (int i = threadIdx.x; i < ntok * HD / 8; i += G * 32) {
      reinterpret_cast<uint4*>(Ks)[i] = ksrc[i];
      reinterpret_cast<uint4*>(Vs)[i] = vsrc[i];
    }
    __syncthreads();
#pragma unroll
    for (int qi = 0; qi < QT; ++qi) {
      if (qi >= nq) continue;
      const int kv_len = pos0 + t0 + qi + 1;              // causal: query t sees positions <= pos0 + t
      const int vis = min(ntok, kv_len - pg * PAGE);
      if (vis <= 0) continue;
#pragma unroll 1
      for (int h0 = 0; h0 < vis; h0 += 32) {
        const int nt = min(32, vis - h0);
        float sc[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          sc[j] = 0.f;
          if (j < nt) {
            const uint2 u = *reinterpret_cast<const uint2*>(Ks + (h0 + j) * HD + lane * 4);
            sc[j] = fmaf(qv[qi][0], bf_lo(u.x), fmaf(qv[qi][1], bf_hi(u.x), fmaf(qv[qi][2], bf_lo(u.y), qv[qi][3] * bf_hi(u.y))));
          }
        }
        transpose_reduce32(sc, lane);
        const bool valid = lane < nt;
        const float s = valid ? sc[0] : -INFINITY;
        const float m_new = fmaxf(m[qi], warp_max(s));
        const float pj = valid ? exp2f((s - m_new) * LOG2E) : 0.f;
        const float corr = exp2f((m[qi] - m_new) * LOG2E);
        l[qi] = l[qi] * corr + warp_sum(pj);
#pragma unroll
        for (int dd = 0; dd < 4; ++dd) o[qi][dd] *= corr;
        m[qi] = m_new;
        ps[warp][lane] = pj;
        __syncwarp();
        for (int j = 0; j < nt; ++j) {
          const float pw = ps[warp][j];
          const uint2 u = *reinterpret_cast<const uint2*>(Vs + (h0 + j) * HD + lane * 4);
          o[qi][0] = fmaf(pw, bf_lo(u.x), o[qi][0]); o[qi][1] = fmaf(pw, bf_hi(u.x), o[qi][1]);
          o[qi][2] = fmaf(pw, bf_lo(u.y), o[qi][2]); o[qi][3] = fmaf(pw, bf_hi(u.y), o[qi][3]);
        }
        __syncwarp();
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int qi = 0; qi < QT; ++qi) {
    if (qi >= nq) continue;
    const float invL = 1.0f / l[qi];
    __align__(8) bf16 ob[4];
#pragma unroll
    for (int dd = 0; dd < 4; ++dd) ob[dd] = __float2bfloat16_rn(o[qi][dd] * invL);
    *reinterpret_cast<uint2*>(out + (size_t)(t0 + qi) * n_heads * HD + head * HD + lane * 4) = *reinterpret_cast<const uint2*>(ob);
  }
}

}  // namespace dn
