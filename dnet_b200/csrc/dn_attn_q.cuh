// dn_attn_q.cuh -- causal attention of a prefill chunk over the 8- / 4-bit quantised KV cache (dn_kvquant.cuh has the format and the
// semantics) on the 5th-generation tensor cores, libdnet_b200.so.
//
// Rows and row blocks are those of k_attn_prefill_tc (dn_attn_tc.cuh), the cluster's share of the keys is attn_q_cut's.  The semantics round scores and
// probabilities to bf16, which an online softmax cannot reproduce: the key tiles are walked twice, first for every row's maximum and
// sum, then for the probabilities and the output.  Rounded numbers land on the other side of an edge by as little as their sums are off, so that
// the sums are kept as short and as small as the format allows.  With codes less the middle of their range (c' = c - 128 or c - 8, exact in bf16)
// and b' = bias + middle x scale,
//   s = scale_0 (Q'_0 c'_0) + scale_1 (Q'_1 c'_1) + b'_0 sum(q'_0) + b'_1 sum(q'_1)      (two groups of 64 dims: an accumulator each, four products
//       long; scales and biases in fp32 by the row's thread)
//   o = sum over tiles of P (hi + lo) + (sum_j p_j b'_0j, sum_j p_j b'_1j)      (scale x c' has at most 16 mantissa bits: hi + lo holds it exactly; P is
//       bf16 by definition; a tile's product and its bias terms join fp32 sums of the row's thread)
// Eight warps turn a tile's codes into operands.
//
// Bound by shared memory: a thread reads sixteen bytes of scales and biases a key in each walk, 262 KB a tile and walk of the 128 bytes a cycle that operands and conversion
// share, and the softmax warps, which form every score twice.  In the first walk the scores have two places, so that a tile's are formed while the other's are read; in the
// second the probabilities have two, and a tile's product joins the sums while the next one's probabilities are formed; codes are asked for a unit ahead.  777 tokens
// behind 1,024 (8 x 4 heads, 8 bits): 237 us with a thread a row, whose one warp a scheduler waits for itself, 190 with two, 161 so; 1,500 behind 3,000 754 and 625; one
// token behind 8,000 90 and 86 before (traced).  (Code units asked for ahead alone, or the two walks' loops rolled: nothing.  With hi + lo keys of scale x code in one
// accumulator of 16 products, and one output accumulator over all
// tiles: 240 and 82.  Of the stored results 1.56 % and 2.64 % then were not the nearest to 64 bits; now 0.19 % and 0.17 %; k_attn_q, whose
// block per (head, token) takes 4.1 ms and 1.4 ms, 0.26 % and 0.66 %.)
// Roles: warp 0 MMA issuer, warp 1 TMEM allocator, warps 4-11 softmax (a thread a row and half of its keys), warps 12-19 conversion.
#pragma once
#include "dn_attn_tc.cuh"
#include "dn_kvquant.cuh"

namespace dn {

struct AqParams {
  AtParams a;
  const unsigned char* pool;     // this layer's packed pages
  int whole;                     // beside a.share: AqCut::whole
};

// How a launch's work is cut: Z CTAs share a row block's keys; with `whole`, each of a key head's `whole` longest row blocks (an even number) is one CTA's
// and only the others are shared.  The CTAs of a launch, longest first, run in rounds of as many as the SMs hold at once; whoever ends first in a round begins first
// in the next, so that a round's last goes with the next one's first.  Taken is what makes the sum of the rounds smallest, in key tiles (6.9 us each) and 1.5 to 2.5
// for a CTA's start, exchange and end (weights and the three tiles that halves behind whole blocks are charged: what is taken is then, on average, within 0.1 % of
// the fastest of all cuts over 380 shapes of 1 to 2,000 tokens behind 0 to 16,000, groups of 1, 4, 5 and 8, and nowhere slower than by the rule of
// k_attn_prefill_tc, whose tiles take a third as long beside the same start and end: 3.7 % less on average).  8 bits, groups of 4, in us by that rule and so: 8 heads, 777
// tokens behind 1,024, 200 blocks in rounds of 148 and 52: 159 and 148; one token behind 500 35 and 25; 300 behind 4,000 243 and 212; 160 behind 8,000 234 and
// 203; 2 heads, 1,500 tokens 90 and 54.
struct AqCut {
  int Z, whole;
};
__host__ __device__ inline AqCut attn_q_cut(int n_kv, int blocks, int tb, int kv_len, int sms) {
  const int n = n_kv * blocks, tiles = (kv_len + 127) / 128, keys = tiles * 128;
  // tenths of a key tile that a CTA of the i-th longest block takes
  auto weight = [&](int i, int Z) {
    const int t = (keys - i / n_kv * tb + 127) / 128;
    return (t + Z - 1) / Z * 10 + (Z == 1 ? 15 : Z == 2 ? 22 : Z == 4 ? 24 : 25);
  };
  auto cost = [&](int Z, int whole) {
    const int at_once = Z == 1 ? sms : Z == 2 ? sms / 2 : Z == 4 ? sms * 33 / 148 : sms * 15 / 148, first = whole * n_kv;
    const int r1 = (first + sms - 1) / sms, rounds = r1 + (n - first + at_once - 1) / at_once;
    int sum = 0;
    for (int r = 0; r < rounds; ++r) {
      const bool end = !(r & 1) && r + 1 < rounds;      // this round's last counts, else its first
      if (r < r1) sum += weight(end ? ((r + 1) * sms < first ? (r + 1) * sms : first) - 1 : r * sms, 1);
      else sum += weight(end ? ((r - r1 + 1) * at_once < n - first ? first + (r - r1 + 1) * at_once : n) - 1 : first + (r - r1) * at_once, Z);
    }
    const int longest = weight(0, whole ? 1 : Z);
    return (sum > longest ? sum : longest) + (whole ? 30 : 0);      // (halves behind whole blocks: their rounds end further apart)
  };
  AqCut best{1, 0};
  int least = cost(1, 0);
  for (int Z = 2; Z <= AT_MAX_Z && tiles >= 2 * Z; Z *= 2) {
    const int c = cost(Z, 0);
    if (c < least) { least = c; best = AqCut{Z, 0}; }
  }
  for (int r = 1; r * sms < n && tiles >= 4; ++r) {      // whole rounds of whole blocks, the others in halves
    const int whole = r * sms / n_kv & ~1, c = whole ? cost(2, whole) : least;
    if (c < least) { least = c; best = AqCut{2, whole}; }
  }
  return best;
}
// a captured launch's clusters (as attn_prefill_split_max)
static inline int attn_q_cut_max(int n_kv, int blocks, int tb, int kv_len, int sms) {
  int best = 1;
  for (int n = (blocks - 1) * tb + 1; n < kv_len + 128 && best < AT_MAX_Z; n += 128) {
    const int z = attn_q_cut(n_kv, blocks, tb, n, sms).Z;
    if (z > best) best = z;
  }
  return best;
}
constexpr int AQT_THREADS = 640, AQT_DQ = 256;
constexpr int AQT_KB = 6 * 128;      // floats of a key tile: scales of both groups, biases of both groups, (bias of group 0, of group 1) of each value row
constexpr int AQT_XCH = (4 * AQT_KB + 2 * AT_MAX_Z * 2 * 128 + 2 * 128) * 4;      // four key tiles' scales and biases, the maxima and sums of both halves of every rank,
                                                                                 // the halves' bias terms
constexpr int AQT_SMEM = 5 * AT_TILE + AQT_XCH + 1024 + 256;
constexpr int AQT_REGS_MMA = 40, AQT_REGS_SOFTMAX = 136, AQT_REGS_DQ = 80;      // setmaxnreg: of the 96 a thread that 640 threads are launched with
static_assert(128 * (AQT_REGS_MMA + 2 * AQT_REGS_SOFTMAX + 2 * AQT_REGS_DQ) <= AQT_THREADS * 96, "setmaxnreg split exceeds the CTA's launch allocation");

template <int G, int BITS>
__global__ void __launch_bounds__(AQT_THREADS, 1) k_attn_prefill_q(const AqParams pq) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int TB = 128 / G;
  constexpr float MID = (float)(1 << (BITS - 1));      // what is taken off the codes
  const AtParams& p = pq.a;
  extern __shared__ __align__(1024) unsigned char tc_smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char *sQ = smem, *sK = smem + AT_TILE, *sV = smem + 3 * AT_TILE;      // K: two tiles in turn; V: hi tile, lo tile
  float* kb = reinterpret_cast<float*>(smem + 5 * AT_TILE);                      // [4][scale 0, scale 1, bias 0, bias 1, value biases (two)][128 keys]
  float* zx = kb + 4 * AQT_KB;                                // [Z][2 halves][2][128]
  float* obx = zx + 2 * AT_MAX_Z * 256;                                          // [2][128]
  float* zo = reinterpret_cast<float*>(sK);                                      // [Z][128 / Z][128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 5 * AT_TILE + AQT_XCH);
  uint64_t *k_full = bars, *k_empty = bars + 2, *v_full = bars + 4, *v_empty = bars + 5, *s_full = bars + 6, *s_empty = bars + 8, *p_full = bars + 10, *o_free = bars + 12,
           *w_full = bars + 13, *w_empty = bars + 17;      // (w: the first walk's scores, [buffer][half])
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 21);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pos0 = p.st->pos, blocks = (p.T + TB - 1) / TB;
  const AqCut cut = p.share > 0 ? AqCut{p.share, pq.whole} : attn_q_cut((int)gridDim.x, blocks, TB, pos0 + p.T, p.sms);
  // a cluster's block, the longest first: whole ones by twos, one each for the cluster's first two CTAs (the others, as all beyond the share, have nothing to do)
  const bool alone = 2 * (int)blockIdx.y < cut.whole;
  const int block = alone ? 2 * (int)blockIdx.y + min((int)blockIdx.z, 1) : (int)blockIdx.y + cut.whole / 2;
  if (block >= blocks) return;
  const int kvh = blockIdx.x, t0 = (blocks - 1 - block) * TB, z = alone && blockIdx.z == 1 ? 0 : (int)blockIdx.z, Z = alone ? 1 : cut.Z;
  const int nq = min(TB, p.T - t0);
  const int kv_max = pos0 + t0 + nq;
  const int pages = (kv_max + PAGE - 1) / PAGE, all = (kv_max + 127) >> 7;
  const int j0 = (int)((long long)all * z / Z), n_tiles = z < Z ? (int)((long long)all * (z + 1) / Z) - j0 : 0;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) { mbar_init(&k_full[i], AQT_DQ / 32); mbar_init(&k_empty[i], 1); mbar_init(&s_full[i], 1); mbar_init(&s_empty[i], 4); }
    mbar_init(v_full, AQT_DQ / 32); mbar_init(v_empty, 1); mbar_init(&p_full[0], 8); mbar_init(&p_full[1], 8); mbar_init(o_free, 8);
    for (int i = 0; i < 4; ++i) { mbar_init(&w_full[i], 1); mbar_init(&w_empty[i], 4); }
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
  // S: two halves of a tile, each 64 keys of group 0, then of group 1 (in the first walk two tiles in turn, the second one's in the columns of P and O); P, two in turn;
  // the tile's product
  const uint32_t tmem = *tmem_slot, tO = tmem + 256, tP = tmem + 384;

  if (warp < 4) {
    // ===================== products =====================
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(AQT_REGS_MMA));
    const uint32_t idesc_s = tc_instr_desc(128, 64), idesc_o = tc_instr_desc(128, 128) | (1u << 16);
    auto scores = [&](int it, uint32_t at, uint64_t* full, uint64_t* empty, uint32_t empty_phase) {      // of the it-th tile of both walks
      const int kbuf = it & 1;
      mbar_wait(&k_full[kbuf], (uint32_t)(it >> 1) & 1u, p.err);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        mbar_wait(&empty[h], empty_phase, p.err);
        tc_fence_after();
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          const uint64_t adesc = tc_smem_desc(sQ + g * 16384), bdesc = tc_smem_desc(sK + kbuf * AT_TILE + g * 16384 + h * 8192);
#pragma unroll
          for (int k = 0; k < 4; ++k) tc_mma(at + h * 128 + g * 64, adesc + (uint64_t)(2 * k), bdesc + (uint64_t)(2 * k), idesc_s, k ? 1u : 0u);
        }
        if (h == 1) tc_commit(&k_empty[kbuf]);
        tc_commit(&full[h]);
      }
    };
    auto scores2 = [&](int j) { scores(n_tiles + j, tmem, s_full, s_empty, ((uint32_t)j & 1u) ^ 1u); };
    if (warp == 0 && lane == 0) {
#pragma unroll 1
      for (int j = 0; j < n_tiles; ++j) scores(j, tmem + (j & 1) * 256, w_full + (j & 1) * 2, w_empty + (j & 1) * 2, ((uint32_t)(j >> 1) & 1u) ^ 1u);
    }
    __syncwarp();
    if (Z > 1) cluster_sync();
    if (warp == 0 && lane == 0) {
      if (n_tiles > 0) {
        const uint32_t uses = (uint32_t)(n_tiles + 1) / 2;      // of the first buffer, which has been read
        mbar_wait(&w_empty[0], (uses - 1) & 1u, p.err);
        mbar_wait(&w_empty[1], (uses - 1) & 1u, p.err);
        scores2(0);
      }
#pragma unroll 1
      for (int j = 0; j < n_tiles; ++j) {
        if (j + 1 < n_tiles) scores2(j + 1);
        mbar_wait(v_full, (uint32_t)j & 1u, p.err);
        mbar_wait(&p_full[j & 1], (uint32_t)(j >> 1) & 1u, p.err);
        mbar_wait(o_free, ((uint32_t)j & 1u) ^ 1u, p.err);
        tc_fence_after();
#pragma unroll
        for (int part = 1; part >= 0; --part) {      // the small part first: fewer sums are cut at the size of the result
          const uint64_t vdesc = tc_smem_desc_mn(sV + part * AT_TILE, 16384, 1024);
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            tc_mma_ts(tO, tP + (j & 1) * 64 + 8 * kk, vdesc + (uint64_t)(kk * (2048 >> 4)), idesc_o, (part == 0 || kk) ? 1u : 0u);
        }
        tc_commit(v_empty);
      }
    }
    __syncwarp();
    if (Z > 1) { cluster_sync(); cluster_sync(); }
  } else if (warp < 12) {
    // ===================== softmax: warps 4-7 take the first half of every tile's keys, warps 8-11 the second, a thread a row =====================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(AQT_REGS_SOFTMAX));
    const int h = (warp - 4) >> 2, qd = warp & 3, r = qd * 32 + lane;      // half of the keys, and of the output's columns; TMEM lane quarter, this thread's row
    const int rg = r / TB, rt = r % TB;
    const bool ok = rg < G && rt < nq;
    const int last = ok ? pos0 + t0 + rt : -1;        // last visible key position
    const uint32_t lane_off = (uint32_t)(qd * 32) << 16;
    float sq0 = 0.f, sq1 = 0.f, m = -INFINITY, l = 0.f, ob0 = 0.f, ob1 = 0.f;
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      const uint4 v = *reinterpret_cast<const uint4*>(sQ + at_swz(r, c));
      const float f = ((bf_lo(v.x) + bf_hi(v.x)) + (bf_lo(v.y) + bf_hi(v.y))) + ((bf_lo(v.z) + bf_hi(v.z)) + (bf_lo(v.w) + bf_hi(v.w)));
      if (c < 8) sq0 += f; else sq1 += f;
    }
    // Sixteen keys of the half tile at a time (900 cycles; eight took 530): the products of both groups into the scores
    // rounded to bf16; keys that the row does not see: -inf.  it, j: the tile, c: 0, 16, 32, 48
    auto scores_of = [&](uint32_t at, int it, int j, int c, float2 (&s)[8]) {
      uint32_t a[16], b[16];
      tm_ld16(at + lane_off + c, a);
      tm_ld16(at + 64 + lane_off + c, b);
      const float4* kf = reinterpret_cast<const float4*>(kb + (it & 3) * AQT_KB + h * 64 + c);
      const int key = ((j0 + j) << 7) + h * 64 + c;
      tm_wait_ld();
      tm_pin16(a);
      tm_pin16(b);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 s0 = kf[i], s1 = kf[32 + i], b0 = kf[64 + i], b1 = kf[96 + i];
        auto two = [&](int e, float2 c0, float2 c1, float2 d0, float2 d1) {
          const float2 x = f2_fma(make_float2(__uint_as_float(a[e]), __uint_as_float(a[e + 1])), c0,
                                  f2_fma(make_float2(__uint_as_float(b[e]), __uint_as_float(b[e + 1])), c1, f2_fma(d0, f2_of(sq0), f2_mul(d1, f2_of(sq1)))));
          const uint32_t w = pack_bf16x2(x.x, x.y);
          s[e / 2] = make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
        };
        two(4 * i, make_float2(s0.x, s0.y), make_float2(s1.x, s1.y), make_float2(b0.x, b0.y), make_float2(b1.x, b1.y));
        two(4 * i + 2, make_float2(s0.z, s0.w), make_float2(s1.z, s1.w), make_float2(b0.z, b0.w), make_float2(b1.z, b1.w));
      }
      if (!__all_sync(0xffffffffu, !ok || key + 15 <= last)) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (key + 2 * i > last) s[i].x = -INFINITY;
          if (key + 2 * i + 1 > last) s[i].y = -INFINITY;
        }
      }
    };
    // ---- first walk: maxima and sums
#pragma unroll 1
    for (int j = 0; j < n_tiles; ++j) {
      // (the key scales were written before the products that these barriers count were issued; their places are used again four tiles later)
      const int w = (j & 1) * 2 + h;
      mbar_wait(&w_full[w], (uint32_t)(j >> 1) & 1u, p.err);
      __syncwarp();
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < 64; c += 16) {
        float2 s[8];
        scores_of(tmem + (j & 1) * 256 + h * 128, j, j, c, s);
        float2 x2 = make_float2(fmaxf(s[0].x, s[1].x), fmaxf(s[0].y, s[1].y)), x3 = make_float2(fmaxf(s[2].x, s[3].x), fmaxf(s[2].y, s[3].y));
#pragma unroll
        for (int i = 4; i < 8; i += 2) {
          x2 = make_float2(fmaxf(x2.x, s[i].x), fmaxf(x2.y, s[i].y));
          x3 = make_float2(fmaxf(x3.x, s[i + 1].x), fmaxf(x3.y, s[i + 1].y));
        }
        const float mx = fmaxf(m, fmaxf(fmaxf(x2.x, x2.y), fmaxf(x3.x, x3.y)));
        const float at = mx == -INFINITY ? 0.f : mx;      // (a row that has seen nothing yet adds zeros)
        float2 e2 = f2_of(0.f), e3 = e2;
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
          const float2 x = f2_mul(f2_add(s[i], f2_of(-at)), f2_of(LOG2E)), y = f2_mul(f2_add(s[i + 1], f2_of(-at)), f2_of(LOG2E));
          e2 = f2_add(e2, make_float2(tc_ex2(x.x), tc_ex2(x.y)));
          e3 = f2_add(e3, make_float2(tc_ex2(y.x), tc_ex2(y.y)));
        }
        e2 = f2_add(e2, e3);
        l = fmaf(l, tc_ex2((m - at) * LOG2E), e2.x + e2.y);
        m = mx;
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&w_empty[w]);
    }
    // the other half's keys count too, and the other ranks'
    if (Z > 1) {
      __syncwarp();
      for (int d = 0; d < (z < Z ? Z : 0); ++d) {
        dsmem_st(dsmem_addr(zx + (z * 2 + h) * 256 + r, (uint32_t)d), m);
        dsmem_st(dsmem_addr(zx + (z * 2 + h) * 256 + 128 + r, (uint32_t)d), l);
      }
      __syncwarp();
      cluster_sync();
    } else {
      zx[h * 256 + r] = m;
      zx[h * 256 + 128 + r] = l;
      asm volatile("bar.sync 1, 256;" ::: "memory");
    }
    {
      float M = -INFINITY, L = 0.f;
      for (int d = 0; d < 2 * Z; ++d) M = fmaxf(M, zx[d * 256 + r]);
      for (int d = 0; d < 2 * Z; ++d) {
        const float mm = zx[d * 256 + r];
        if (mm != -INFINITY) L += exp2f((mm - M) * LOG2E) * zx[d * 256 + 128 + r];
      }
      m = M;
      l = L;
    }
    // ---- second walk: probabilities and output
    const float inv = 1.0f / l;
    float o[64];      // columns 64 h ..
#pragma unroll
    for (int i = 0; i < 64; ++i) o[i] = 0.f;
    auto join = [&](int j) {      // the j-th tile's product joins the row's sums
      mbar_wait(v_empty, (uint32_t)j & 1u, p.err);
      __syncwarp();
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t a[32];
        tm_ld32(tO + lane_off + h * 64 + c * 32, a);
        tm_wait_ld();
        tm_pin(a);
#pragma unroll
        for (int i = 0; i < 32; ++i) o[c * 32 + i] += __uint_as_float(a[i]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(o_free);
    };
#pragma unroll 1
    for (int j = 0; j < n_tiles; ++j) {
      const int it = n_tiles + j;
      float2 t0s = f2_of(0.f), t1s = t0s;
      mbar_wait(&s_full[h], (uint32_t)j & 1u, p.err);
      __syncwarp();
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < 64; c += 16) {
        float2 s[8];
        scores_of(tmem + h * 128, it, j, c, s);
        const float4* b4 = reinterpret_cast<const float4*>(kb + (it & 3) * AQT_KB + 512) + (h * 64 + c) / 2;
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float2 x = f2_mul(f2_add(s[i], f2_of(-m)), f2_of(LOG2E)), e = f2_mul(make_float2(tc_ex2(x.x), tc_ex2(x.y)), f2_of(inv));
          w[i] = ok ? pack_bf16x2(e.x, e.y) : 0u;
          const float pa = __uint_as_float(w[i] << 16), pd = __uint_as_float(w[i] & 0xffff0000u);
          const float4 bv = b4[i];
          t0s = f2_fma(f2_of(pa), make_float2(bv.x, bv.y), t0s);
          t1s = f2_fma(f2_of(pd), make_float2(bv.z, bv.w), t1s);
        }
        tm_st8(tP + (j & 1) * 64 + lane_off + h * 32 + c / 2, w);      // (the product that read this one's place was joined a tile ago)
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_empty[h]);
      ob0 += t0s.x + t1s.x;
      ob1 += t0s.y + t1s.y;
      tm_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[j & 1]);
      if (j > 0) join(j - 1);      // (formed while this tile's probabilities were)
    }
    if (n_tiles > 0) join(n_tiles - 1);
    // the bias terms of both halves' keys: this thread's columns are those of group h
    obx[h * 128 + r] = h ? ob0 : ob1;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    const float ob = h ? obx[r] + ob1 : ob0 + obx[128 + r];
#pragma unroll
    for (int i = 0; i < 64; ++i) o[i] += n_tiles > 0 ? ob : 0.f;
    __syncwarp();
    if (Z > 1) cluster_sync();      // every rank's products are done: its key buffers may take the other ranks' columns
    const int per = 128 / Z, lg = 31 - __clz(per);      // columns of a rank: a power of two
    if (Z > 1) {
      if (z < Z)
#pragma unroll
        for (int i = 0; i < 64; ++i) dsmem_st(dsmem_addr(zo + (z * per + ((h * 64 + i) & (per - 1))) * 128 + r, (uint32_t)((h * 64 + i) >> lg)), o[i]);
      __syncwarp();
      cluster_sync();
      if (ok && z < Z) {
        bf16* dst = p.out + ((size_t)(t0 + rt) * p.n_heads + kvh * G + rg) * HD + z * per;
        for (int c = h * (per / 2); c < (h + 1) * (per / 2); c += 8) {
          float y[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) y[i] = 0.f;
          for (int d = 0; d < Z; ++d)
#pragma unroll
            for (int i = 0; i < 8; ++i) y[i] += zo[((size_t)d * per + c + i) * 128 + r];
          *reinterpret_cast<uint4*>(dst + c) = make_uint4(pack_bf16x2(y[0], y[1]), pack_bf16x2(y[2], y[3]), pack_bf16x2(y[4], y[5]), pack_bf16x2(y[6], y[7]));
        }
      }
    } else if (ok && z == 0) {
      bf16* dst = p.out + ((size_t)(t0 + rt) * p.n_heads + kvh * G + rg) * HD + h * 64;
#pragma unroll
      for (int k = 0; k < 8; ++k)
        *reinterpret_cast<uint4*>(dst + k * 8) = make_uint4(pack_bf16x2(o[8 * k], o[8 * k + 1]), pack_bf16x2(o[8 * k + 2], o[8 * k + 3]),
                                                           pack_bf16x2(o[8 * k + 4], o[8 * k + 5]), pack_bf16x2(o[8 * k + 6], o[8 * k + 7]));
    }
  } else {
    // ===================== codes into operands =====================
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(AQT_REGS_DQ));
    constexpr int CH = KvQ<BITS>::ROW_BYTES / 16, PER = 128 * CH / AQT_DQ;      // 16-byte chunks of a row, of a thread
    constexpr int CODES = 128 / BITS;                                           // codes of a chunk: 16 / 32
    const int dt = (int)threadIdx.x - (AQT_THREADS - AQT_DQ);
    // The codes, less MID, of eight numbers, the o-th eight of the chunk: a code as the low byte of 2^23 + code, one subtraction for two
    auto codes8 = [&](const uint4& cw, int o, float2 (&f)[4]) {
      const uint32_t u[4] = {cw.x, cw.y, cw.z, cw.w};
      const float2 off = f2_of(-(8388608.f + MID));
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint32_t a, b;
        if (BITS == 8) {
          const uint32_t w = u[(o * 2 + (k >> 1)) & 3];
          a = __byte_perm(w, 0x4B000000u, 0x7440 + (k & 1) * 2);
          b = __byte_perm(w, 0x4B000000u, 0x7441 + (k & 1) * 2);
        } else {
          a = __byte_perm(u[o & 3] & 0x0f0f0f0fu, 0x4B000000u, 0x7440 + k);
          b = __byte_perm((u[o & 3] >> 4) & 0x0f0f0f0fu, 0x4B000000u, 0x7440 + k);
        }
        f[k] = f2_add(f2_bits(a, b), off);
      }
    };
    // A unit is a tile's keys or values: those of the first walk, then keys and values of the second in turn.  The next unit's codes are on their way while one is
    // turned into operands.
    // codes; keys: scales and biases of row dt (threads 0 .. 127; 128 .. 255: of the second walk's value rows); values: the scale of each chunk's row and group
    struct Unit { uint4 cw[PER]; uint32_t sw, bw; uint32_t sc[PER]; };
    const int units = 3 * n_tiles;
    auto tile_of = [&](int x) { return x < n_tiles ? x : (x - n_tiles) >> 1; };
    auto load = [&](int x, Unit& U) {
      const int j = tile_of(x), kv = x >= n_tiles ? (x - n_tiles) & 1 : 0, key0 = (j0 + j) << 7, pl = 2 * (j0 + j);
      const int pg0 = p.block_table[pl], pg1 = pl + 1 < pages ? p.block_table[pl + 1] : pg0;
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int y = i * AQT_DQ + dt, row = y / CH, c = y % CH;
        const unsigned char* unit = kvq_unit<BITS>(pq.pool, row < 64 ? pg0 : pg1, kv, kvh, p.n_kv);
        const bool have = key0 + row < kv_max;      // rows that belong to no key: whatever the page holds, it must not enter
        U.cw[i] = have ? __ldcg(reinterpret_cast<const uint4*>(unit + (size_t)(row & 63) * KvQ<BITS>::ROW_BYTES) + c) : make_uint4(0u, 0u, 0u, 0u);
        U.sc[i] = kv && have ? (uint32_t)__ldcg(reinterpret_cast<const unsigned short*>(unit + KvQ<BITS>::CODES_BYTES) + (row & 63) * 2 + (c * CODES >= 64 ? 1 : 0)) : 0u;
      }
      U.sw = U.bw = 0u;
      if (!kv && key0 + (dt & 127) < kv_max && (dt < 128 || x >= n_tiles)) {
        const uint32_t* sb = reinterpret_cast<const uint32_t*>(kvq_unit<BITS>(pq.pool, (dt & 127) < 64 ? pg0 : pg1, dt >> 7, kvh, p.n_kv) + KvQ<BITS>::CODES_BYTES);
        U.sw = __ldcg(sb + (dt & 63));
        U.bw = __ldcg(sb + PAGE + (dt & 63));
      }
    };
    auto keys = [&](int it, const Unit& U) {
      unsigned char* dst = sK + (it & 1) * AT_TILE;
      mbar_wait(&k_empty[it & 1], ((uint32_t)(it >> 1) & 1u) ^ 1u, p.err);
      if (dt < 128) {
        float* f = kb + (it & 3) * AQT_KB + dt;
        f[0] = bf_lo(U.sw); f[128] = bf_hi(U.sw);
        f[256] = fmaf(bf_lo(U.sw), MID, bf_lo(U.bw)); f[384] = fmaf(bf_hi(U.sw), MID, bf_hi(U.bw));
      } else if (it >= n_tiles)
        *reinterpret_cast<float2*>(kb + (it & 3) * AQT_KB + 512 + 2 * (dt - 128)) = make_float2(fmaf(bf_lo(U.sw), MID, bf_lo(U.bw)), fmaf(bf_hi(U.sw), MID, bf_hi(U.bw)));
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int x = i * AQT_DQ + dt, row = x / CH, c = x % CH;
#pragma unroll
        for (int o = 0; o < CODES / 8; ++o) {       // eight codes: a 16-byte chunk of the tile
          float2 f[4];
          codes8(U.cw[i], o, f);
          *reinterpret_cast<uint4*>(dst + at_swz(row, c * (CODES / 8) + o)) =
              make_uint4(upper_halves(f[0].x, f[0].y), upper_halves(f[1].x, f[1].y), upper_halves(f[2].x, f[2].y), upper_halves(f[3].x, f[3].y));      // (exact: eight bits)
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&k_full[it & 1]);
    };
    auto values = [&](int j, const Unit& U) {
      mbar_wait(v_empty, ((uint32_t)j & 1u) ^ 1u, p.err);
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int x = i * AQT_DQ + dt, row = x / CH, c = x % CH;
        const float2 sc = f2_of(__uint_as_float(U.sc[i] << 16));
#pragma unroll
        for (int o = 0; o < CODES / 8; ++o) {       // eight codes: one 16-byte chunk of each tile
          float2 f[4];
          codes8(U.cw[i], o, f);
          uint32_t hi[4], lo[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float2 y = f2_mul(f[k], sc);
            hi[k] = pack_bf16x2(y.x, y.y);
            const float2 r = f2_fma(f2_bits(hi[k] << 16, hi[k] & 0xffff0000u), f2_of(-1.f), y);
            lo[k] = pack_bf16x2(r.x, r.y);
          }
          const uint32_t at = at_swz(row, c * (CODES / 8) + o);
          *reinterpret_cast<uint4*>(sV + at) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
          *reinterpret_cast<uint4*>(sV + AT_TILE + at) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(v_full);
    };
    Unit cur, nxt;
    if (units > 0) load(0, cur);
#pragma unroll 1
    for (int x = 0; x < units; ++x) {
      if (x + 1 < units) load(x + 1, nxt);
      if (x < n_tiles) keys(x, cur);
      else if (((x - n_tiles) & 1) == 0) keys(n_tiles + tile_of(x), cur);
      else values(tile_of(x), cur);
      cur = nxt;
      if (x == n_tiles - 1) { __syncwarp(); if (Z > 1) cluster_sync(); }      // (the end of the first walk)
    }
    if (units == 0) { __syncwarp(); if (Z > 1) cluster_sync(); }
    __syncwarp();
    if (Z > 1) { cluster_sync(); cluster_sync(); }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
}

}  // namespace dn
