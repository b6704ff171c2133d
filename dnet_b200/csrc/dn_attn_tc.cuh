// dn_attn_tc.cuh -- causal attention of a prefill chunk over the paged 16-bit KV cache on the 5th-generation tensor cores
// (tcgen05 + TMEM + TMA), libdnet_b200.so.
//
// Chunks of few row blocks, whose keys several CTAs share; those of many run on k_attn_prompt (dn_attn_prompt.cuh, attn_prompt_from).
//
// A CTA takes one key / value head, its G query heads and TB = floor(128 / G) consecutive query tokens: the 128 MMA rows are heads
// x tokens (row = g TB + t), so that a staged key / value tile serves the whole group; with G = 5 or 7 a few rows stay empty.  The
// key tiles (128 keys, two pages, by TMA through the block table) go in turn to two sides, each with its own running reference,
// sums and output: while the weights of one side's tile are formed, the tensor cores run the other's products.  Per tile:
//   S = Q K^T       A = Q [128 x 128], B = K tile [128 x 128], both K-major in shared memory      TMEM columns 128 side ..
//   P = weights     four warps a side, a thread a row: 2^(score - reference); P takes the place of S in TMEM: of each 32 columns
//                   the first 16 hold 32 weights as bf16, the other 16 what bf16 left of them (16 bits of each weight's mantissa);
//                   what those two leave (all 24 bits) has 64 columns of its own                      TMEM columns 384 + 64 side ..
//   P V             A = P out of TMEM, B = V tile, MN-major, the small parts first
//                   TMEM columns 256 + 128 side .. with two parts; with three, 256 .. of both sides in turn
// The row's thread adds the tile's product to its own 128 fp32 sums, which it scales when the running maximum (the reference) moves: in TMEM the
// accumulator is cut, not rounded, at every 16 keys.  The scores are read twice, for the maximum and for the weights: sums and scores do not
// fit into one thread's registers.  At the end the two sides meet in TMEM.
// Long contexts and few query tokens: the Z CTAs of a cluster take a share of the key tiles each and add their outputs through
// distributed shared memory, every CTA the columns of 128 / Z dims.
//
// Bound by the softmax warps (some six instructions and an exponential a score) beside the products (1,536 cycles a tile with two
// parts, 2,048 with three).  Measured, 512 tokens behind 8,192: eight groups of 4 heads 109 us with two parts, 148 with three; eight groups of 5
// 234 with two CTAs a cluster (what attn_prefill_split takes), 269 with four; 2,048 tokens, groups of 4: 90 us.  With one accumulator over all
// tiles of a side, and two parts for every group, they were 98, 168, 207 and 80; error against 64 bits before the result is stored, groups of 5
// behind 8,192 / 300: 5.3e-6 / 2.2e-6 so, 3.0e-7 / 2.6e-7 now, 1.6e-6 / 3.6e-7 on the CUDA cores; groups of 4 behind 8,192 with two parts: 2.6e-6 / 2.1e-6.
// Roles: warp 0 TMA producer, warp 1 MMA issuer, warp 2 TMEM allocator, warps 4-7 side 0, warps 8-11 side 1.
#pragma once
#include "dn_gemm_tc.cuh"

namespace dn {

// 8 and 16 consecutive 32-bit columns of this warp's TMEM quarter
__device__ __forceinline__ void tm_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
// 16 columns; valid after tm_wait_ld and tm_pin16
__device__ __forceinline__ void tm_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
                 "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr));
}
__device__ __forceinline__ void tm_pin16(uint32_t (&r)[16]) {
#pragma unroll
  for (int i = 0; i < 16; i += 8)
    asm volatile("" : "+r"(r[i]), "+r"(r[i + 1]), "+r"(r[i + 2]), "+r"(r[i + 3]), "+r"(r[i + 4]), "+r"(r[i + 5]), "+r"(r[i + 6]), "+r"(r[i + 7]));
}

struct AtParams {
  const bf16* q;                 // [T][n_heads][128] (RoPE applied, unscaled)
  bf16* out;                     // [T][n_heads][128]
  const int32_t* block_table;
  const StepState* st;
  int n_heads, n_kv, T;
  int share, sms;                // CTAs of a cluster that take keys (0: by the position in the step state)
  unsigned int* err;
};

constexpr int AT_TILE = 128 * 128 * 2;     // one [128 x 128] bf16 tile = 32 KiB (two 64-column halves)
constexpr int AT_MAX_Z = 8;                // CTAs of a cluster that share a row block's keys
constexpr int AT_XCH = (4 * 128 + AT_MAX_Z * 2 * 128) * 4;      // the sides' references and sums; every cluster rank's
constexpr int AT_SMEM = 5 * AT_TILE + AT_XCH + 1024 + 256;
constexpr int AT_THREADS = 384;
// A weight is held in two bf16 parts (16 bits of its mantissa; 2^-18 of it at most is lost) or three (all 24).  Three take a third more products.
// Chunks of fewer tokens than this and groups of 5 and 7 take them: they are as close to 64 bits as fp32 weights on the CUDA cores are (see above;
// single tokens behind 256 / 8,192: 2.7e-7 / 2.9e-7, k_attn 2.0e-7 / 4.7e-7).  (Chunks whose group has up to FEW_ROWS rows run on k_attn_few.)
constexpr int AT_TWO_PARTS_FROM = 16;
static inline int attn_parts(int G, int T) { return G == 5 || G == 7 || (G >= 4 && T < AT_TWO_PARTS_FROM) ? 3 : 2; }
constexpr int AT_REGS_MMA = 56, AT_REGS_SOFTMAX = 224;      // setmaxnreg: of the 168 a thread that 384 threads are launched with
static_assert(128 * AT_REGS_MMA + 256 * AT_REGS_SOFTMAX <= AT_THREADS * 168, "setmaxnreg split exceeds the CTA's launch allocation");

// CTAs that share a row block's keys: what makes (waves of CTAs) x (key tiles of a CTA + 4 for its start, joining and end) smallest.
// The grid alone (heads x row blocks) leaves most SMs idle when a chunk is short, and a last wave nearly empty when it is long:
// 40 heads in groups of 5, 512 tokens give 168 CTAs for 148 SMs.
// Of 148 SMs 74 clusters of two run at once, 33 of four and 15 of eight (what tc_clusters is answered on this board; held here as constants, since the kernel
// itself counts when it replays a captured chunk: a board whose processing clusters are cut otherwise gets the same results, perhaps later): behind 8,192 tokens these 168 row blocks take 234 us with
// Z = 2 and 269 with 4, which a count that takes every SM for usable by every cluster prefers (a layer 798 us so, 770 now).
__host__ __device__ inline int attn_prefill_split(int ctas, int kv_len, int sms) {
  const int tiles = (kv_len + 127) / 128;
  int best = 1, cost = 0;
  for (int Z = 1; Z <= AT_MAX_Z; Z *= 2) {
    if (Z > 1 && tiles < 2 * Z) break;
    const int at_once = Z == 1 ? sms : Z == 2 ? sms / 2 : Z == 4 ? sms * 33 / 148 : sms * 15 / 148;
    const int c = ((ctas + at_once - 1) / at_once) * ((tiles + Z - 1) / Z + (Z > 1 ? 6 : 4));
    if (Z == 1 || c < cost) { cost = c; best = Z; }
  }
  return best;
}

// A captured launch is replayed at positions that nobody knows yet: its clusters are as large as the longest share needs, the kernel takes the
// share of the position it finds (AtParams::share 0), and the CTAs beyond it stay idle -- the sums of a replay are those of an eager launch.
static inline int attn_prefill_split_max(int ctas, int kv_len, int sms) {
  int best = 1;
  for (int n = 128; n < kv_len + 128 && best < AT_MAX_Z; n += 128) {
    const int z = attn_prefill_split(ctas, n, sms);
    if (z > best) best = z;
  }
  return best;
}

// two fp32 operations, each rounded as the single one
__device__ __forceinline__ float2 f2_mul(float2 a, float2 b) {
  float2 r;
  asm("{.reg .b64 x, y, z; mov.b64 x, {%2, %3}; mov.b64 y, {%4, %5}; mul.rn.f32x2 z, x, y; mov.b64 {%0, %1}, z;}" : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 f2_add(float2 a, float2 b) {
  float2 r;
  asm("{.reg .b64 x, y, z; mov.b64 x, {%2, %3}; mov.b64 y, {%4, %5}; add.rn.f32x2 z, x, y; mov.b64 {%0, %1}, z;}" : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 f2_fma(float2 a, float2 b, float2 c) {
  float2 r;
  asm("{.reg .b64 x, y, z, w; mov.b64 x, {%2, %3}; mov.b64 y, {%4, %5}; mov.b64 z, {%6, %7}; fma.rn.f32x2 w, x, y, z; mov.b64 {%0, %1}, w;}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}
__device__ __forceinline__ float2 f2_of(float x) { return make_float2(x, x); }
// two numbers cut to bf16, and what is cut off
__device__ __forceinline__ uint32_t upper_halves(float a, float b) { return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632); }
__device__ __forceinline__ float2 below_upper_halves(float2 a) {
  return f2_fma(make_float2(__uint_as_float(__float_as_uint(a.x) & 0xffff0000u), __uint_as_float(__float_as_uint(a.y) & 0xffff0000u)), f2_of(-1.f), a);
}
__device__ __forceinline__ float2 f2_bits(uint32_t a, uint32_t b) { return make_float2(__uint_as_float(a), __uint_as_float(b)); }
__device__ __forceinline__ void tm_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
        "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

template <int G, int PARTS>
__global__ void __launch_bounds__(AT_THREADS, 1) k_attn_prefill_tc(const __grid_constant__ CUtensorMap mapKV, const AtParams p) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int TB = 128 / G;
  extern __shared__ __align__(1024) unsigned char tc_smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char *sQ = smem, *sK = smem + AT_TILE, *sV = smem + 3 * AT_TILE;      // K and V: one buffer a side
  float* xch = reinterpret_cast<float*>(smem + 5 * AT_TILE);                     // [2][128] references, [2][128] sums of the sides
  float* zx = xch + 512;                                                         // [Z][2][128]: every rank's reference and sum
  float* zo = reinterpret_cast<float*>(sK);                                      // [Z][128 / Z][128]: every rank's output columns
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 5 * AT_TILE + AT_XCH);
  uint64_t *k_full = bars, *k_empty = bars + 2, *v_full = bars + 4, *v_empty = bars + 6, *s_full = bars + 8, *p_full = bars + 10, *o_full = bars + 12, *o_free = bars + 14;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // (the cluster spans the grid's z; the row blocks with the most keys start first, so that the last to run are short)
  const int kvh = blockIdx.x, t0 = (int)(gridDim.y - 1 - blockIdx.y) * TB, z = blockIdx.z;
  const int pos0 = p.st->pos;
  const int Z = p.share > 0 ? p.share : attn_prefill_split((int)(gridDim.x * gridDim.y), pos0 + p.T, p.sms);      // ranks from Z on have no keys and no columns
  const int nq = min(TB, p.T - t0);                         // query tokens of this CTA
  const int kv_max = pos0 + t0 + nq;                        // keys visible to its last query
  const int pages = (kv_max + PAGE - 1) / PAGE, all = (kv_max + 127) >> 7;
  const int j0 = (int)((long long)all * z / Z), n_tiles = z < Z ? (int)((long long)all * (z + 1) / Z) - j0 : 0;      // this CTA's key tiles

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 4); mbar_init(&o_full[i], 1);
    }
    mbar_init(o_free, 4);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // Q tile: rows (g, t) <- q[t0 + t][kvh*G + g][:], zero rows where there is none; written with the TMA 128B swizzle
  for (int i = threadIdx.x; i < 128 * 16; i += AT_THREADS) {
    const int r = i >> 4, c = i & 15;
    const int g = r / TB, t = r % TB;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (g < G && t < nq) v = *reinterpret_cast<const uint4*>(p.q + ((size_t)(t0 + t) * p.n_heads + kvh * G + g) * HD + c * 8);
    *reinterpret_cast<uint4*>(sQ + at_swz(r, c)) = v;
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // generic-proxy writes -> visible to the MMA (async proxy)
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot, tO = tmem + 256;

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(AT_REGS_MMA));      // a softmax thread holds its row's 128 sums
    if (warp == 0 && lane == 0) {
      for (int j = 0; j < n_tiles; ++j) {
        const int sd = j & 1;
        const uint32_t ph = (uint32_t)(j >> 1) & 1u;
        const int pl = 2 * (j0 + j);
        const int pg0 = p.block_table[pl], pg1 = pl + 1 < pages ? p.block_table[pl + 1] : pg0;      // an unused half: any valid page (masked)
        const int rk0 = ((pg0 * 2 + 0) * p.n_kv + kvh) * PAGE, rk1 = ((pg1 * 2 + 0) * p.n_kv + kvh) * PAGE;
        const int rv0 = ((pg0 * 2 + 1) * p.n_kv + kvh) * PAGE, rv1 = ((pg1 * 2 + 1) * p.n_kv + kvh) * PAGE;
        unsigned char *dk = sK + sd * AT_TILE, *dv = sV + sd * AT_TILE;
        mbar_wait(&k_empty[sd], ph ^ 1u, p.err);
        mbar_arrive_expect_tx(&k_full[sd], AT_TILE);
        tma_load_2d(dk, &mapKV, 0, rk0, &k_full[sd]);
        tma_load_2d(dk + 16384, &mapKV, 64, rk0, &k_full[sd]);
        tma_load_2d(dk + 8192, &mapKV, 0, rk1, &k_full[sd]);
        tma_load_2d(dk + 16384 + 8192, &mapKV, 64, rk1, &k_full[sd]);
        mbar_wait(&v_empty[sd], ph ^ 1u, p.err);
        mbar_arrive_expect_tx(&v_full[sd], AT_TILE);
        tma_load_2d(dv, &mapKV, 0, rv0, &v_full[sd]);
        tma_load_2d(dv + 16384, &mapKV, 64, rv0, &v_full[sd]);
        tma_load_2d(dv + 8192, &mapKV, 0, rv1, &v_full[sd]);
        tma_load_2d(dv + 16384 + 8192, &mapKV, 64, rv1, &v_full[sd]);
      }
    }
    if (warp == 1 && lane == 0) {
      const uint32_t idesc_s = tc_instr_desc(128, 128);
      const uint32_t idesc_o = tc_instr_desc(128, 128) | (1u << 16);       // V is MN-major
      auto scores = [&](int j) {
        const int sd = j & 1;
        mbar_wait(&k_full[sd], (uint32_t)(j >> 1) & 1u, p.err);
        tc_fence_after();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint64_t adesc = tc_smem_desc(sQ + h * 16384), bdesc = tc_smem_desc(sK + sd * AT_TILE + h * 16384);
#pragma unroll
          for (int k = 0; k < 4; ++k) tc_mma(tmem + sd * 128, adesc + (uint64_t)(2 * k), bdesc + (uint64_t)(2 * k), idesc_s, (h | k) ? 1u : 0u);
        }
        tc_commit(&k_empty[sd]);
        tc_commit(&s_full[sd]);
      };
      if (n_tiles > 0) scores(0);
      if (n_tiles > 1) scores(1);
      for (int j = 0; j < n_tiles; ++j) {
        const int sd = j & 1;
        const uint32_t ph = (uint32_t)(j >> 1) & 1u;
        mbar_wait(&v_full[sd], ph, p.err);
        mbar_wait(&p_full[sd], ph, p.err);
        if (PARTS == 3 && j > 0) mbar_wait(o_free, (uint32_t)(j - 1) & 1u, p.err);      // the other side has read its product
        tc_fence_after();
        const uint64_t vdesc = tc_smem_desc_mn(sV + sd * AT_TILE, 16384, 1024);
#pragma unroll
        for (int part = PARTS - 1; part >= 0; --part)      // the small parts first: fewer sums are cut at the size of the result
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            tc_mma_ts(tO + (PARTS == 2 ? sd * 128 : 0), part == 2 ? tmem + 384 + sd * 64 + 8 * kk : tmem + sd * 128 + 32 * (kk >> 1) + 8 * (kk & 1) + 16 * part,
                      vdesc + (uint64_t)(kk * (2048 >> 4)), idesc_o, (part < PARTS - 1 || kk) ? 1u : 0u);
        tc_commit(&v_empty[sd]);
        tc_commit(&o_full[sd]);
        if (j + 2 < n_tiles) scores(j + 2);      // into the columns that P has just been read from: products run in order
      }
    }
    __syncwarp();
    if (Z > 1) { cluster_sync(); cluster_sync(); }      // (the other warps' below)
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(AT_REGS_SOFTMAX));
    const int sd = (warp - 4) >> 2, qd = warp & 3, r = qd * 32 + lane;      // side, TMEM lane quarter, this thread's row
    const int g = r / TB, t = r % TB;
    const bool ok = g < G && t < nq;
    const int pos = pos0 + t0 + t;                     // last visible key position (causal)
    const int last = ok ? pos : -1;
    const uint32_t lane_off = (uint32_t)(qd * 32) << 16, tS = tmem + sd * 128 + lane_off, tOs = tO + (PARTS == 2 ? sd * 128 : 0) + lane_off;
    const float sc2 = 0.08838834764831845f * LOG2E;
    float ref = -INFINITY, l = 0.f;      // ref: scaled, log2
    float2 o[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) o[i] = f2_of(0.f);
    for (int j = sd; j < n_tiles; j += 2) {
      const uint32_t ph = (uint32_t)(j >> 1) & 1u;
      const int key0 = (j0 + j) << 7;
      mbar_wait(&s_full[sd], ph, p.err);
      __syncwarp();
      tc_fence_after();
      // every key of the tile is seen by every live row of the warp (rows without a query compute something that is not stored)
      const bool all_seen = __all_sync(0xffffffffu, !ok || key0 + 127 <= pos);
      auto unseen = [&](int c, uint32_t (&v)[32]) {      // of 32 columns, those of keys that the row does not see: -inf
        tm_pin(v);
        if (!all_seen) {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (key0 + c * 32 + i > last) v[i] = 0xff800000u;
        }
      };
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < 4; c += 2) {
        uint32_t a[32], b[32];
        tm_ld32(tS + c * 32, a);
        tm_ld32(tS + c * 32 + 32, b);
        tm_wait_ld();
        unseen(c, a);
        unseen(c + 1, b);
#pragma unroll
        for (int i = 0; i < 32; ++i) mx[i & 3] = fmaxf(fmaxf(mx[i & 3], __uint_as_float(a[i])), __uint_as_float(b[i]));      // (one instruction)
      }
      const float ref_new = fmaxf(ref, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * sc2);
      const float f = ref == ref_new ? 1.f : exp2f(ref - ref_new);      // 0 for a row that has seen nothing yet
      ref = ref_new;
      const float nref = ref == -INFINITY ? 0.f : -ref;
      float2 l0 = f2_of(0.f), l1 = l0;
      uint32_t va[2][32];
      tm_ld32(tS, va[0]);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t (&v)[32] = va[c & 1];
        uint32_t w[32], x[16];
        tm_wait_ld();
        unseen(c, v);
        if (c < 3) tm_ld32(tS + c * 32 + 32, va[(c + 1) & 1]);      // on its way while this one's weights are formed
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float2 y = f2_fma(f2_bits(v[2 * i], v[2 * i + 1]), f2_of(sc2), f2_of(nref));
          float2 e = make_float2(tc_ex2(y.x), tc_ex2(y.y));
          if (i & 1) l1 = f2_add(l1, e); else l0 = f2_add(l0, e);
          if (PARTS == 3) {      // cut, not rounded: three times eight bits hold all 24
            w[i] = upper_halves(e.x, e.y);
            e = below_upper_halves(e);
            w[16 + i] = upper_halves(e.x, e.y);
            e = below_upper_halves(e);
            x[i] = upper_halves(e.x, e.y);
          } else {
            w[i] = pack_bf16x2(e.x, e.y);
            e = f2_fma(f2_bits(w[i] << 16, w[i] & 0xffff0000u), f2_of(-1.f), e);
            w[16 + i] = pack_bf16x2(e.x, e.y);
          }
        }
        tmem_st32(tS + c * 32, w);
        if (PARTS == 3) tm_st16(tmem + 384 + sd * 64 + lane_off + c * 16, x);
      }
      l0 = f2_add(l0, l1);
      l = fmaf(l, f, l0.x + l0.y);
      if (key0 + 128 > kv_max) {      // value rows that belong to no key: whatever the page holds, it must not enter
        const int valid = kv_max - key0;
        mbar_wait(&v_full[sd], ph, p.err);
        for (int i = threadIdx.x - 128 - sd * 128; i < (128 - valid) * 16; i += 128) {
          const int row = valid + (i >> 4), c = i & 15;
          *reinterpret_cast<uint4*>(sV + sd * AT_TILE + (c >> 3) * 16384 + row * 128 + (c & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      }
      tm_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[sd]);
      // the tile's product joins the row's sums
      mbar_wait(&o_full[sd], ph, p.err);
      __syncwarp();
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 4; c += 2) {
        uint32_t a[32], b[32];
        tm_ld32(tOs + c * 32, a);
        tm_ld32(tOs + c * 32 + 32, b);
        tm_wait_ld();
        tm_pin(a);
        tm_pin(b);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          o[c * 16 + i] = f2_fma(o[c * 16 + i], f2_of(f), f2_bits(a[2 * i], a[2 * i + 1]));
          o[c * 16 + 16 + i] = f2_fma(o[c * 16 + 16 + i], f2_of(f), f2_bits(b[2 * i], b[2 * i + 1]));
        }
      }
      if (PARTS == 3) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(o_free);
      }
    }
    // the two sides meet in TMEM: no product is under way any more and every side has read its last one
    tc_fence_before();
    asm volatile("bar.sync 1, 256;" ::: "memory");
    tc_fence_after();
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint32_t v[32];
#pragma unroll
      for (int i = 0; i < 16; ++i) { v[2 * i] = __float_as_uint(o[c * 16 + i].x); v[2 * i + 1] = __float_as_uint(o[c * 16 + i].y); }
      tmem_st32(tO + sd * 128 + lane_off + c * 32, v);
    }
    tm_wait_st();
    xch[sd * 128 + r] = ref;
    xch[256 + sd * 128 + r] = l;
    tc_fence_before();
    __syncwarp();
    if (Z > 1) cluster_sync();      // every CTA's products are done: its key buffers may take the other ranks' columns
    asm volatile("bar.sync 1, 256;" ::: "memory");
    tc_fence_after();
    // the thread's row, half of its columns: both sides' outputs relative to the larger reference
    const float r0 = xch[r], r1 = xch[128 + r], M = fmaxf(r0, r1);
    const float f0 = r0 == -INFINITY ? 0.f : exp2f(r0 - M), f1 = r1 == -INFINITY ? 0.f : exp2f(r1 - M);
    const float L = f0 * xch[256 + r] + f1 * xch[384 + r];
    float y[64];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      uint32_t a[32], b[32];
      tm_ld32(tO + lane_off + sd * 64 + c * 32, a);
      tm_ld32(tO + lane_off + 128 + sd * 64 + c * 32, b);
      tm_wait_ld();
      tm_pin(a);
      tm_pin(b);
#pragma unroll
      for (int i = 0; i < 32; ++i) y[c * 32 + i] = f0 * __uint_as_float(a[i]) + f1 * __uint_as_float(b[i]);
    }
    if (Z == 1) {
      if (ok && z == 0) {
        const float inv = 1.0f / L;
        bf16* dst = p.out + ((size_t)(t0 + t) * p.n_heads + kvh * G + g) * HD + sd * 64;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          uint4 w;
          w.x = pack_bf16x2(y[8 * c] * inv, y[8 * c + 1] * inv); w.y = pack_bf16x2(y[8 * c + 2] * inv, y[8 * c + 3] * inv);
          w.z = pack_bf16x2(y[8 * c + 4] * inv, y[8 * c + 5] * inv); w.w = pack_bf16x2(y[8 * c + 6] * inv, y[8 * c + 7] * inv);
          *reinterpret_cast<uint4*>(dst + c * 8) = w;
        }
      }
    } else if (z < Z) {
      const int per = 128 / Z;      // columns of a rank
#pragma unroll
      for (int i = 0; i < 64; ++i) {
        const int col = sd * 64 + i, dst = col / per;
        dsmem_st(dsmem_addr(zo + ((size_t)z * per + col % per) * 128 + r, (uint32_t)dst), y[i]);
      }
      if (sd == 0)
        for (int d = 0; d < Z; ++d) {
          dsmem_st(dsmem_addr(zx + z * 256 + r, (uint32_t)d), M);
          dsmem_st(dsmem_addr(zx + z * 256 + 128 + r, (uint32_t)d), L);
        }
    }
    tc_fence_before();
    if (Z > 1) {
      __syncwarp();
      cluster_sync();
      if (ok && z < Z) {
        const int per = 128 / Z, half = per / 2;
        float M = -INFINITY, L = 0.f;
        for (int d = 0; d < Z; ++d) M = fmaxf(M, zx[d * 256 + r]);
        for (int d = 0; d < Z; ++d) {
          const float m = zx[d * 256 + r];
          if (m != -INFINITY) L += exp2f(m - M) * zx[d * 256 + 128 + r];
        }
        const float inv = 1.0f / L;
        bf16* dst = p.out + ((size_t)(t0 + t) * p.n_heads + kvh * G + g) * HD + z * per + sd * half;
        for (int c = 0; c < half; c += 8) {
          float q8[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) q8[i] = 0.f;
          for (int d = 0; d < Z; ++d) {
            const float m = zx[d * 256 + r], f = m == -INFINITY ? 0.f : exp2f(m - M);
#pragma unroll
            for (int i = 0; i < 8; ++i) q8[i] = fmaf(f, zo[((size_t)d * per + sd * half + c + i) * 128 + r], q8[i]);
          }
          uint4 w;
          w.x = pack_bf16x2(q8[0] * inv, q8[1] * inv); w.y = pack_bf16x2(q8[2] * inv, q8[3] * inv);
          w.z = pack_bf16x2(q8[4] * inv, q8[5] * inv); w.w = pack_bf16x2(q8[6] * inv, q8[7] * inv);
          *reinterpret_cast<uint4*>(dst + c) = w;
        }
      }
    }
  }
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
}

}  // namespace dn
