// dn_attn_tc.cuh -- causal attention of a prefill chunk over the paged 16-bit KV cache on the 5th-generation tensor cores
// (tcgen05 + TMEM + TMA), libdnet_b200.so.
//
// A CTA takes one key / value head, its G query heads and TB = floor(128 / G) consecutive query tokens: the 128 MMA rows are heads
// x tokens (row = g TB + t), so that a staged key / value tile serves the whole group; with G = 5 or 7 a few rows stay empty.  The
// key tiles (128 keys, two pages, by TMA through the block table) go in turn to two sides, each with its own running reference,
// sums and output: while the weights of one side's tile are formed, the tensor cores run the other's products.  Per tile:
//   S = Q K^T       A = Q [128 x 128], B = K tile [128 x 128], both K-major in shared memory      TMEM columns 128 side ..
//   P = weights     four warps a side, a thread a row: 2^(score - reference); P takes the place of S in TMEM: of each 32 columns
//                   the first 16 hold 32 weights as bf16, the other 16 what bf16 left of them (16 bits of each weight's mantissa:
//                   the probabilities stay as good as fp32 against the bf16 values they multiply)
//   O += P V        A = P out of TMEM, B = V tile, MN-major                                      TMEM columns 256 + 128 side ..
// The reference is a running maximum that moves (and O is scaled by the row's own thread) only when a score exceeds it by 2^8, so
// that scaling is rare and every sum stays in range.  At the end the two sides meet in shared memory.
// Long contexts and few query tokens: the Z CTAs of a cluster take a share of the key tiles each and add their outputs through
// distributed shared memory, every CTA the columns of 128 / Z dims.
//
// Bound by the tensor cores (three 128 x 128 x 128 products a tile, 1,536 cycles) with the exponentials (1,024 cycles of the special
// function units) beside them.  Measured: 512 tokens behind 8,192 of a Qwen2.5-32B layer (groups of 5), whole layer 7,205 -> 1,037 us
// (the CUDA-core kernel took 6,400); a Llama-3-8B prompt of 2,048 tokens, two layers and head, 4,154 -> 3,901 us (one side, one
// buffer, P through shared memory before).
// Roles: warp 0 TMA producer, warp 1 MMA issuer, warp 2 TMEM allocator, warps 4-7 side 0, warps 8-11 side 1.
#pragma once
#include "dn_gemm_tc.cuh"

namespace dn {

struct AtParams {
  const bf16* q;                 // [T][n_heads][128] (RoPE applied, unscaled)
  bf16* out;                     // [T][n_heads][128]
  const int32_t* block_table;
  const StepState* st;
  int n_heads, n_kv, T;
  unsigned int* err;
};

constexpr int AT_TILE = 128 * 128 * 2;     // one [128 x 128] bf16 tile = 32 KiB (two 64-column halves)
constexpr int AT_MAX_Z = 8;                // CTAs of a cluster that share a row block's keys
constexpr int AT_XCH = (4 * 128 + AT_MAX_Z * 2 * 128) * 4;      // the sides' references and sums; every cluster rank's
constexpr int AT_SMEM = 5 * AT_TILE + AT_XCH + 1024 + 256;
constexpr int AT_THREADS = 384;
constexpr float AT_SLACK = 8.f;            // how far (log2) a score may exceed the reference before the row is rescaled

template <int G>
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
  uint64_t *k_full = bars, *k_empty = bars + 2, *v_full = bars + 4, *v_empty = bars + 6, *s_full = bars + 8, *p_full = bars + 10, *o_full = bars + 12;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 13);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kvh = blockIdx.x, t0 = blockIdx.y * TB, Z = gridDim.z, z = blockIdx.z;      // the cluster spans the grid's z
  const int pos0 = p.st->pos;
  const int nq = min(TB, p.T - t0);                         // query tokens of this CTA
  const int kv_max = pos0 + t0 + nq;                        // keys visible to its last query
  const int pages = (kv_max + PAGE - 1) / PAGE, all = (kv_max + 127) >> 7;
  const int j0 = (int)((long long)all * z / Z), n_tiles = (int)((long long)all * (z + 1) / Z) - j0;      // this CTA's key tiles

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 4);
    }
    mbar_init(o_full, 1);
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

  if (warp == 0) {
    if (lane == 0) {
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
  } else if (warp == 1) {
    if (lane == 0) {
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
        tc_fence_after();
        const uint64_t vdesc = tc_smem_desc_mn(sV + sd * AT_TILE, 16384, 1024);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
#pragma unroll
          for (int part = 0; part < 2; ++part)
            tc_mma_ts(tO + sd * 128, tmem + sd * 128 + 32 * (kk >> 1) + 8 * (kk & 1) + 16 * part, vdesc + (uint64_t)(kk * (2048 >> 4)), idesc_o,
                      (j > 1 || kk || part) ? 1u : 0u);
        }
        tc_commit(&v_empty[sd]);
        if (j + 2 < n_tiles) scores(j + 2);      // into the columns that P has just been read from: products run in order
      }
      tc_commit(o_full);
    }
  } else if (warp >= 4) {
    const int sd = (warp - 4) >> 2, qd = warp & 3, r = qd * 32 + lane;      // side, TMEM lane quarter, this thread's row
    const int g = r / TB, t = r % TB;
    const bool ok = g < G && t < nq;
    const int pos = pos0 + t0 + t;                     // last visible key position (causal)
    const uint32_t lane_off = (uint32_t)(qd * 32) << 16, tS = tmem + sd * 128 + lane_off, tOs = tO + sd * 128 + lane_off;
    const float sc2 = 0.08838834764831845f * LOG2E;
    float ref = -INFINITY, l = 0.f;      // ref: scaled, log2
    for (int j = sd; j < n_tiles; j += 2) {
      const uint32_t ph = (uint32_t)(j >> 1) & 1u;
      const int key0 = (j0 + j) << 7;
      uint32_t v[4][32];
      mbar_wait(&s_full[sd], ph, p.err);
      __syncwarp();
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 4; ++c) tm_ld32(tS + c * 32, v[c]);
      tm_wait_ld();
#pragma unroll
      for (int c = 0; c < 4; ++c) tm_pin(v[c]);
      // every key of the tile is seen by every live row of the warp (rows without a query compute something that is not stored)
      if (!__all_sync(0xffffffffu, !ok || key0 + 127 <= pos)) {
        const int last = ok ? pos : -1;
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (key0 + c * 32 + i > last) v[c][i] = 0xff800000u;      // -inf
      }
      float mx = -INFINITY;
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int i = 0; i < 32; ++i) mx = fmaxf(mx, __uint_as_float(v[c][i]));
      mx *= sc2;
      const bool move = mx > ref + AT_SLACK || (ref == -INFINITY && mx > -INFINITY);
      if (__any_sync(0xffffffffu, move)) {
        const float f = move ? exp2f(ref - mx) : 1.f;      // 0 for a row that has seen nothing yet
        if (move) { ref = mx; l *= f; }
        if (j > 1) {      // (the side's previous product with V is complete: its scores were issued behind it)
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t o[32];
            tm_ld32(tOs + c * 32, o);
            tm_wait_ld();
            tm_pin(o);
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
            tmem_st32(tOs + c * 32, o);
          }
        }
      }
      const float nref = ref == -INFINITY ? 0.f : -ref;
      float l0 = 0.f, l1 = 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t w[32];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float a = tc_ex2(fmaf(__uint_as_float(v[c][2 * i]), sc2, nref)), d = tc_ex2(fmaf(__uint_as_float(v[c][2 * i + 1]), sc2, nref));
          l0 += a; l1 += d;
          w[i] = pack_bf16x2(a, d);
          w[16 + i] = pack_bf16x2(a - __uint_as_float(w[i] << 16), d - __uint_as_float(w[i] & 0xffff0000u));
        }
        tmem_st32(tS + c * 32, w);
      }
      l += l0 + l1;
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
    }
    xch[sd * 128 + r] = ref;
    xch[256 + sd * 128 + r] = l;
    mbar_wait(o_full, 0u, p.err);
    __syncwarp();
    tc_fence_after();
  }
  __syncwarp();
  if (Z > 1) cluster_sync();      // every CTA's products are done: its key buffers may take the other ranks' columns
  if (warp >= 4) {
    asm volatile("bar.sync 1, 256;" ::: "memory");
    const int sd = (warp - 4) >> 2, qd = warp & 3, r = qd * 32 + lane;
    const int g = r / TB, t = r % TB;
    const bool ok = g < G && t < nq;
    const uint32_t lane_off = (uint32_t)(qd * 32) << 16;
    // the thread's row, half of its columns: both sides' outputs relative to the larger reference
    const float r0 = xch[r], r1 = xch[128 + r], M = fmaxf(r0, r1);
    const float f0 = r0 == -INFINITY ? 0.f : exp2f(r0 - M), f1 = r1 == -INFINITY ? 0.f : exp2f(r1 - M);
    const float L = f0 * xch[256 + r] + f1 * xch[384 + r];
    float o[64];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      uint32_t a[32], b[32];
      if (n_tiles > 0) tm_ld32(tO + lane_off + sd * 64 + c * 32, a);
      if (n_tiles > 1) tm_ld32(tO + lane_off + 128 + sd * 64 + c * 32, b);
      tm_wait_ld();
      tm_pin(a);
      tm_pin(b);
#pragma unroll
      for (int i = 0; i < 32; ++i)      // (a side without a tile has not written its columns)
        o[c * 32 + i] = (n_tiles > 0 ? f0 * __uint_as_float(a[i]) : 0.f) + (n_tiles > 1 ? f1 * __uint_as_float(b[i]) : 0.f);
    }
    if (Z == 1) {
      if (ok) {
        const float inv = 1.0f / L;
        bf16* dst = p.out + ((size_t)(t0 + t) * p.n_heads + kvh * G + g) * HD + sd * 64;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          uint4 w;
          w.x = pack_bf16x2(o[8 * c] * inv, o[8 * c + 1] * inv); w.y = pack_bf16x2(o[8 * c + 2] * inv, o[8 * c + 3] * inv);
          w.z = pack_bf16x2(o[8 * c + 4] * inv, o[8 * c + 5] * inv); w.w = pack_bf16x2(o[8 * c + 6] * inv, o[8 * c + 7] * inv);
          *reinterpret_cast<uint4*>(dst + c * 8) = w;
        }
      }
    } else {
      const int per = 128 / Z;      // columns of a rank
#pragma unroll
      for (int i = 0; i < 64; ++i) {
        const int col = sd * 64 + i, dst = col / per;
        dsmem_st(dsmem_addr(zo + ((size_t)z * per + col % per) * 128 + r, (uint32_t)dst), o[i]);
      }
      if (sd == 0)
        for (int d = 0; d < Z; ++d) {
          dsmem_st(dsmem_addr(zx + z * 256 + r, (uint32_t)d), M);
          dsmem_st(dsmem_addr(zx + z * 256 + 128 + r, (uint32_t)d), L);
        }
    }
    tc_fence_before();
  }
  if (Z > 1) {
    __syncwarp();
    cluster_sync();
    if (warp >= 4) {
      const int sd = (warp - 4) >> 2, r = (warp & 3) * 32 + lane;
      const int g = r / TB, t = r % TB;
      if (g < G && t < nq) {
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
          float o[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = 0.f;
          for (int d = 0; d < Z; ++d) {
            const float m = zx[d * 256 + r], f = m == -INFINITY ? 0.f : exp2f(m - M);
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = fmaf(f, zo[((size_t)d * per + sd * half + c + i) * 128 + r], o[i]);
          }
          uint4 w;
          w.x = pack_bf16x2(o[0] * inv, o[1] * inv); w.y = pack_bf16x2(o[2] * inv, o[3] * inv);
          w.z = pack_bf16x2(o[4] * inv, o[5] * inv); w.w = pack_bf16x2(o[6] * inv, o[7] * inv);
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

// CTAs that share a row block's keys: what makes (waves of CTAs) x (key tiles of a CTA + 4 for its start, joining and end) smallest.
// The grid alone (heads x row blocks) leaves most SMs idle when a chunk is short, and a last wave nearly empty when it is long:
// 40 heads in groups of 5, 512 tokens give 168 CTAs for 148 SMs.
static inline int attn_prefill_split(int ctas, int kv_len, int sms) {
  const int tiles = (kv_len + 127) / 128;
  int best = 1;
  long long cost = 0;
  for (int Z = 1; Z <= AT_MAX_Z; Z *= 2) {
    if (Z > 1 && tiles < 2 * Z) break;
    const long long c = (long long)((ctas * Z + sms - 1) / sms) * ((tiles + Z - 1) / Z + (Z > 1 ? 6 : 4));
    if (Z == 1 || c < cost) { cost = c; best = Z; }
  }
  return best;
}

}  // namespace dn
