// dn_attn_q.cuh -- causal attention of a prefill chunk over the 8- / 4-bit quantised KV cache (dn_kvquant.cuh has the format and the
// semantics) on the 5th-generation tensor cores, libdnet_b200.so.
//
// Rows, blocks and the cluster's share of the keys are those of k_attn_prefill_tc (dn_attn_tc.cuh).  The semantics round scores and
// probabilities to bf16, which an online softmax cannot reproduce: the key tiles are walked twice, first for every row's maximum and
// sum, then for the probabilities and the output.  Eight warps turn a tile's codes into operands: scale x code has at most 16 mantissa
// bits, so a pair of bf16 (hi, lo) holds it exactly, and with exact products and fp32 accumulators
//   s = Q' (hi + lo)^T + bias_0 sum(q'_0) + bias_1 sum(q'_1)      (two groups of 64 dims; the bias terms in fp32 by the row's thread)
//   o = P (hi + lo) + (sum_j p_j bias_0j, sum_j p_j bias_1j)      (P is bf16 by definition)
// are the sums that the CUDA-core kernel (k_attn_q) forms, in another order.
//
// Bound by the tensor cores and the dequantising warps alike: a tile of 128 keys takes 1,024 cycles of products in the first walk and
// 2,048 in the second, beside 640 and 1,280 cycles of conversion.  A block per (head, token) on the CUDA cores read every key row once
// per query instead: 777 tokens behind 1,024 of a Llama-3-8B layer took 4.1 ms.
// Roles: warp 0 MMA issuer, warp 1 TMEM allocator, warps 4-7 softmax (a thread a row), warps 8-15 dequantisation.
#pragma once
#include "dn_attn_tc.cuh"
#include "dn_kvquant.cuh"

namespace dn {

struct AqParams {
  AtParams a;
  const unsigned char* pool;     // this layer's packed pages
};
constexpr int AQT_THREADS = 512, AQT_DQ = 256;
constexpr int AQT_XCH = (4 * 128 * 2 + 128 * 2 + AT_MAX_Z * 2 * 128) * 4;      // key biases of four tiles, value biases, the ranks' maxima and sums
constexpr int AQT_SMEM = 5 * AT_TILE + AQT_XCH + 1024 + 256;

template <int G, int BITS>
__global__ void __launch_bounds__(AQT_THREADS, 1) k_attn_prefill_q(const AqParams pq) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int TB = 128 / G;
  const AtParams& p = pq.a;
  extern __shared__ __align__(1024) unsigned char tc_smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char *sQ = smem, *sK = smem + AT_TILE, *sV = smem + 3 * AT_TILE;      // K, V: hi tile, lo tile
  float2* kb = reinterpret_cast<float2*>(smem + 5 * AT_TILE);                    // [4][128]: (bias of group 0, of group 1) of a key row
  float2* vb = kb + 4 * 128;                                                     // [128]
  float* zx = reinterpret_cast<float*>(vb + 128);                                // [Z][2][128]
  float* zo = reinterpret_cast<float*>(sK);                                      // [Z][128 / Z][128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 5 * AT_TILE + AQT_XCH);
  uint64_t *k_full = bars, *k_empty = bars + 1, *v_full = bars + 2, *v_empty = bars + 3, *s_full = bars + 4, *s_empty = bars + 6, *p_full = bars + 8, *o_full = bars + 9;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 10);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kvh = blockIdx.x, t0 = blockIdx.y * TB, Z = gridDim.z, z = blockIdx.z;
  const int pos0 = p.st->pos;
  const int nq = min(TB, p.T - t0);
  const int kv_max = pos0 + t0 + nq;
  const int pages = (kv_max + PAGE - 1) / PAGE, all = (kv_max + 127) >> 7;
  const int j0 = (int)((long long)all * z / Z), n_tiles = (int)((long long)all * (z + 1) / Z) - j0;

  if (threadIdx.x == 0) {
    mbar_init(k_full, AQT_DQ / 32); mbar_init(k_empty, 1); mbar_init(v_full, AQT_DQ / 32); mbar_init(v_empty, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(&s_full[i], 1); mbar_init(&s_empty[i], 4); }
    mbar_init(p_full, 4); mbar_init(o_full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // Q rows (g, t): q' = T(q hd^-1/2), zero rows where there is none
  for (int i = threadIdx.x; i < 128 * 16; i += AQT_THREADS) {
    const int r = i >> 4, c = i & 15;
    const int g = r / TB, t = r % TB;
    __align__(16) bf16 w[8];
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (g < G && t < nq) v = *reinterpret_cast<const uint4*>(p.q + ((size_t)(t0 + t) * p.n_heads + kvh * G + g) * HD + c * 8);
    const float f[8] = {bf_lo(v.x), bf_hi(v.x), bf_lo(v.y), bf_hi(v.y), bf_lo(v.z), bf_hi(v.z), bf_lo(v.w), bf_hi(v.w)};
#pragma unroll
    for (int k = 0; k < 8; ++k) w[k] = __float2bfloat16_rn(__fmul_rn(f[k], 0.08838834764831845f));
    *reinterpret_cast<uint4*>(sQ + at_swz(r, c)) = *reinterpret_cast<const uint4*>(w);
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  if (Z > 1) cluster_sync();      // every CTA of the cluster has started: the first walk's end stores into the others' memory
  tc_fence_after();
  const uint32_t tmem = *tmem_slot, tP = tmem + 256, tO = tmem + 320;      // S in two buffers of 128 columns

  const uint32_t idesc_s = tc_instr_desc(128, 128), idesc_o = tc_instr_desc(128, 128) | (1u << 16);
  // ---- S of the it-th tile of both walks
  auto scores = [&](int it) {
    mbar_wait(k_full, (uint32_t)it & 1u, p.err);
    mbar_wait(&s_empty[it & 1], ((uint32_t)(it >> 1) & 1u) ^ 1u, p.err);
    tc_fence_after();
#pragma unroll
    for (int part = 0; part < 2; ++part)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint64_t adesc = tc_smem_desc(sQ + h * 16384), bdesc = tc_smem_desc(sK + part * AT_TILE + h * 16384);
#pragma unroll
        for (int k = 0; k < 4; ++k) tc_mma(tmem + (it & 1) * 128, adesc + (uint64_t)(2 * k), bdesc + (uint64_t)(2 * k), idesc_s, (part | h | k) ? 1u : 0u);
      }
    tc_commit(k_empty);
    tc_commit(&s_full[it & 1]);
  };
  // ---- one tile's codes into operands.  kv 0: keys, 1: values
  const int dt = (int)threadIdx.x - (AQT_THREADS - AQT_DQ);
  auto dequant = [&](int j, int kv, unsigned char* dst, float2* bias, uint64_t* empty, uint32_t phase, uint64_t* full) {
    constexpr int CH = KvQ<BITS>::ROW_BYTES / 16, PER = 128 * CH / AQT_DQ;      // 16-byte chunks of a row, of a thread
    constexpr int CODES = 128 / BITS;                                           // codes of a chunk: 16 / 32
    const int key0 = (j0 + j) << 7, pl = 2 * (j0 + j);
    const int pg0 = p.block_table[pl], pg1 = pl + 1 < pages ? p.block_table[pl + 1] : pg0;
    uint4 cw[PER];
    float sc[PER];
    float2 bv = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int x = i * AQT_DQ + dt, row = x / CH, c = x % CH;
      const unsigned char* unit = kvq_unit<BITS>(pq.pool, row < 64 ? pg0 : pg1, kv, kvh, p.n_kv);
      const unsigned short* s = reinterpret_cast<const unsigned short*>(unit + KvQ<BITS>::CODES_BYTES);
      const bool live = key0 + row < kv_max;      // rows that belong to no key: whatever the page holds, it must not enter
      cw[i] = live ? __ldcg(reinterpret_cast<const uint4*>(unit + (size_t)(row & 63) * KvQ<BITS>::ROW_BYTES) + c) : make_uint4(0u, 0u, 0u, 0u);
      sc[i] = live ? __uint_as_float((uint32_t)__ldcg(s + (row & 63) * 2 + (c * CODES >= 64 ? 1 : 0)) << 16) : 0.f;
    }
    if (dt < 128 && key0 + dt < kv_max) {
      const unsigned char* unit = kvq_unit<BITS>(pq.pool, dt < 64 ? pg0 : pg1, kv, kvh, p.n_kv);
      const uint32_t b = __ldcg(reinterpret_cast<const uint32_t*>(unit + KvQ<BITS>::CODES_BYTES + PAGE * 4) + (dt & 63));
      bv = make_float2(bf_lo(b), bf_hi(b));
    }
    mbar_wait(empty, phase, p.err);
    if (dt < 128) bias[dt] = bv;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int x = i * AQT_DQ + dt, row = x / CH, c = x % CH;
      const uint32_t u[4] = {cw[i].x, cw[i].y, cw[i].z, cw[i].w};
#pragma unroll
      for (int o = 0; o < CODES / 8; ++o) {       // eight codes: one 16-byte chunk of each tile
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          float a, b;
          if (BITS == 8) {
            const uint32_t w = u[(o * 2 + (k >> 1)) & 3] >> (16 * (k & 1));
            a = (float)(w & 0xffu); b = (float)((w >> 8) & 0xffu);
          } else {
            const uint32_t w = u[o & 3] >> (8 * k);
            a = (float)(w & 0xfu); b = (float)((w >> 4) & 0xfu);
          }
          a *= sc[i]; b *= sc[i];
          hi[k] = pack_bf16x2(a, b);
          lo[k] = pack_bf16x2(a - __uint_as_float(hi[k] << 16), b - __uint_as_float(hi[k] & 0xffff0000u));
        }
        const uint32_t at = at_swz(row, c * (CODES / 8) + o);
        *reinterpret_cast<uint4*>(dst + at) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(dst + AT_TILE + at) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) mbar_arrive(full);
  };

  const int qd = warp & 3, r = qd * 32 + lane;      // softmax: TMEM lane quarter, this thread's row
  const int rg = r / TB, rt = r % TB;
  const bool ok = rg < G && rt < nq;
  const int last = ok ? pos0 + t0 + rt : -1;        // last visible key position
  const uint32_t lane_off = (uint32_t)(qd * 32) << 16;
  float sq0 = 0.f, sq1 = 0.f, m = -INFINITY, l = 0.f, ob0 = 0.f, ob1 = 0.f;
  const bool smx = warp >= 4 && warp < 8;
  if (smx) {
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      const uint4 v = *reinterpret_cast<const uint4*>(sQ + at_swz(r, c));
      const float f = ((bf_lo(v.x) + bf_hi(v.x)) + (bf_lo(v.y) + bf_hi(v.y))) + ((bf_lo(v.z) + bf_hi(v.z)) + (bf_lo(v.w) + bf_hi(v.w)));
      if (c < 8) sq0 += f; else sq1 += f;
    }
  }
  // 32 scores of this row from column c on, rounded to bf16; keys that the row does not see: -inf
  auto load_scores = [&](int it, int j, int c, float (&s)[32]) {
    uint32_t v[32];
    tm_ld32(tmem + (it & 1) * 128 + lane_off + c, v);
    tm_wait_ld();
    tm_pin(v);
    const float4* b4 = reinterpret_cast<const float4*>(kb + (it & 3) * 128 + c);
    const int key = ((j0 + j) << 7) + c;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float4 b = b4[i];
      s[2 * i] = key + 2 * i <= last ? bf16r(fmaf(b.y, sq1, fmaf(b.x, sq0, __uint_as_float(v[2 * i])))) : -INFINITY;
      s[2 * i + 1] = key + 2 * i + 1 <= last ? bf16r(fmaf(b.w, sq1, fmaf(b.z, sq0, __uint_as_float(v[2 * i + 1])))) : -INFINITY;
    }
  };

  // ===================== first walk: maxima and sums =====================
  if (warp == 0) {
    if (lane == 0)
      for (int j = 0; j < n_tiles; ++j) scores(j);
  } else if (smx) {
    for (int j = 0; j < n_tiles; ++j) {
      // (the key biases were written before the products that these barriers count were issued; their places are used again four tiles later)
      mbar_wait(&s_full[j & 1], (uint32_t)(j >> 1) & 1u, p.err);
      __syncwarp();
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < 128; c += 32) {
        float s[32], mx = m;
        load_scores(j, j, c, s);
#pragma unroll
        for (int i = 0; i < 32; ++i) mx = fmaxf(mx, s[i]);
        const float at = mx == -INFINITY ? 0.f : mx;      // (a row that has seen nothing yet adds zeros)
        float a = 0.f;
#pragma unroll
        for (int i = 0; i < 32; ++i) a += tc_ex2((s[i] - at) * LOG2E);
        l = fmaf(l, tc_ex2((m - at) * LOG2E), a);
        m = mx;
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_empty[j & 1]);
    }
  } else if (warp >= 8) {
    for (int j = 0; j < n_tiles; ++j) dequant(j, 0, sK, kb + (j & 3) * 128, k_empty, ((uint32_t)j & 1u) ^ 1u, k_full);
  }
  if (Z > 1) {      // the other ranks' keys count too
    __syncwarp();
    if (smx)
      for (int d = 0; d < Z; ++d) {
        dsmem_st(dsmem_addr(zx + z * 256 + r, (uint32_t)d), m);
        dsmem_st(dsmem_addr(zx + z * 256 + 128 + r, (uint32_t)d), l);
      }
    __syncwarp();
    cluster_sync();
    if (smx) {
      float M = -INFINITY, L = 0.f;
      for (int d = 0; d < Z; ++d) M = fmaxf(M, zx[d * 256 + r]);
      for (int d = 0; d < Z; ++d) {
        const float mm = zx[d * 256 + r];
        if (mm != -INFINITY) L += exp2f((mm - M) * LOG2E) * zx[d * 256 + 128 + r];
      }
      m = M;
      l = L;
    }
  }
  // ===================== second walk: probabilities and output =====================
  if (warp == 0) {
    if (lane == 0) {
      if (n_tiles > 0) scores(n_tiles);
      for (int j = 0; j < n_tiles; ++j) {
        if (j + 1 < n_tiles) scores(n_tiles + j + 1);
        mbar_wait(v_full, (uint32_t)j & 1u, p.err);
        mbar_wait(p_full, (uint32_t)j & 1u, p.err);
        tc_fence_after();
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          const uint64_t vdesc = tc_smem_desc_mn(sV + part * AT_TILE, 16384, 1024);
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            tc_mma_ts(tO, tP + 8 * kk, vdesc + (uint64_t)(kk * (2048 >> 4)), idesc_o, (j | part | kk) ? 1u : 0u);
        }
        tc_commit(v_empty);
      }
      tc_commit(o_full);
    }
  } else if (smx) {
    const float inv = 1.0f / l;
    for (int j = 0; j < n_tiles; ++j) {
      const int it = n_tiles + j;
      mbar_wait(&s_full[it & 1], (uint32_t)(it >> 1) & 1u, p.err);
      mbar_wait(v_full, (uint32_t)j & 1u, p.err);             // the value biases are written
      if (j > 0) mbar_wait(v_empty, (uint32_t)(j - 1) & 1u, p.err);      // the product before has read its probabilities
      __syncwarp();
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < 128; c += 32) {
        float s[32];
        load_scores(it, j, c, s);
        const float4* b4 = reinterpret_cast<const float4*>(vb + c);
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float a = ok ? tc_ex2((s[2 * i] - m) * LOG2E) * inv : 0.f, d = ok ? tc_ex2((s[2 * i + 1] - m) * LOG2E) * inv : 0.f;
          w[i] = pack_bf16x2(a, d);
          const float pa = __uint_as_float(w[i] << 16), pd = __uint_as_float(w[i] & 0xffff0000u);
          const float4 b = b4[i];
          ob0 = fmaf(pa, b.x, fmaf(pd, b.z, ob0));
          ob1 = fmaf(pa, b.y, fmaf(pd, b.w, ob1));
        }
        tm_st16(tP + lane_off + c / 2, w);
      }
      tm_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) { mbar_arrive(&s_empty[it & 1]); mbar_arrive(p_full); }
    }
    mbar_wait(o_full, 0u, p.err);
    __syncwarp();
    tc_fence_after();
  } else if (warp >= 8) {
    for (int j = 0; j < n_tiles; ++j) {
      const int it = n_tiles + j;
      dequant(j, 0, sK, kb + (it & 3) * 128, k_empty, ((uint32_t)it & 1u) ^ 1u, k_full);
      dequant(j, 1, sV, vb, v_empty, ((uint32_t)j & 1u) ^ 1u, v_full);
    }
  }
  __syncwarp();
  if (Z > 1) cluster_sync();      // every rank's products are done: its key buffers may take the other ranks' columns
  if (smx) {
    const int per = 128 / Z;      // columns of a rank
#pragma unroll 1
    for (int c = 0; c < 128; c += 32) {
      uint32_t o[32];
      if (n_tiles > 0) tm_ld32(tO + lane_off + c, o);
      tm_wait_ld();
      tm_pin(o);
      const float ob = c < 64 ? ob0 : ob1;
      float y[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) y[i] = n_tiles > 0 ? __uint_as_float(o[i]) + ob : 0.f;
      if (Z > 1) {
#pragma unroll
        for (int i = 0; i < 32; ++i) dsmem_st(dsmem_addr(zo + ((size_t)z * per + (c + i) % per) * 128 + r, (uint32_t)((c + i) / per)), y[i]);
      } else if (ok) {
        bf16* dst = p.out + ((size_t)(t0 + rt) * p.n_heads + kvh * G + rg) * HD + c;
#pragma unroll
        for (int k = 0; k < 4; ++k)
          *reinterpret_cast<uint4*>(dst + k * 8) = make_uint4(pack_bf16x2(y[8 * k], y[8 * k + 1]), pack_bf16x2(y[8 * k + 2], y[8 * k + 3]),
                                                             pack_bf16x2(y[8 * k + 4], y[8 * k + 5]), pack_bf16x2(y[8 * k + 6], y[8 * k + 7]));
      }
    }
    tc_fence_before();
  }
  if (Z > 1) {
    __syncwarp();
    cluster_sync();
    if (smx && ok) {
      const int per = 128 / Z;
      bf16* dst = p.out + ((size_t)(t0 + rt) * p.n_heads + kvh * G + rg) * HD + z * per;
      for (int c = 0; c < per; c += 8) {
        float y[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) y[i] = 0.f;
        for (int d = 0; d < Z; ++d)
#pragma unroll
          for (int i = 0; i < 8; ++i) y[i] += zo[((size_t)d * per + c + i) * 128 + r];
        *reinterpret_cast<uint4*>(dst + c) = make_uint4(pack_bf16x2(y[0], y[1]), pack_bf16x2(y[2], y[3]), pack_bf16x2(y[4], y[5]), pack_bf16x2(y[6], y[7]));
      }
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
}

}  // namespace dn
