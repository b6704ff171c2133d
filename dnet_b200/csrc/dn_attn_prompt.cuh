// dn_attn_prompt.cuh -- softmax attention of prompt portions over paged 16-bit keys and values on the 5th-generation tensor cores
// (tcgen05 + TMEM + TMA), head size 128; both libraries.
//
// An item is one key / value head, its G query heads and TB = floor(128 / G) consecutive query tokens (row = token x G + head: 128 MMA rows, a staged
// key / value tile serves the whole group) against the keys that these see, in tiles of 128 (two pages, by TMA through the block table).  The grid is a
// CTA an SM, and a CTA takes whole items (dealt out by length) or, where that leaves the CTAs too unequal, an equal run of the line of all items' tiles: items that a run
// cuts are joined by the CTA that finishes last, from partial outputs in global memory, in the order of the keys (an atomic count, nobody waits).  Within a
// share there is no start and no end between tiles, whichever item they belong to:
//   S = Q K^T       A = Q [128 x 128], B = K tile [128 x 128], both K-major in shared memory      TMEM columns 0 ..: SIDES regions in turn
//   P = weights     four warps a side, a thread a row: 2^(score - reference), where the reference is the tile's own maximum, raised to a power of two; P takes
//                   the place of S: of each 16 columns the first 8 hold 16 weights as bf16, the other 8 what bf16 left of them (16 bits of each
//                   weight's mantissa); with three parts what those two leave (all 24 bits) has 64 columns of its own
//   P V             A = P out of TMEM, B = V tile, MN-major, the small parts first               TMEM columns 384 ..
// The eight summing warps add the tile's product, two threads a row, to fp32 sums, scaled by powers of two, which round nothing: in TMEM the accumulator
// is cut, not rounded, at every 16 keys.
// Bound by the products: 24 (32) MMAs a tile of some 80 cycles, not 64, since operands, copies and the other side's products share the memory port, and a wait for the
// summing warps, which have one product region, between a tile's P V and the next: 2,250 cycles a tile with two parts.  The weights' 1,024 cycles of exponentials a
// tile lie beside them.  Loops are kept short: twenty warps in three roles share four instruction caches, and with the weights' loop unrolled (4 x 32 columns, twice)
// a tile took 5,400 cycles, most of them waiting for instructions.  Halves of 64 dims a product, so that one is read while the other is formed, cost as much a MMA as 128.
// Microseconds, k_attn_prefill_tc / this, eight groups of 4: 2,048 tokens 84 / 62; 700 23 / 21; 512 behind 8,192 115 / 103; 1,500 behind 3,000 162 / 134; of 5 (three parts):
// 512 behind 8,192 242 / 160; 1,000 behind 0 52 / 37, behind 4,000 246 / 166; 300 19 / 17.5.
// Roles: warp 0 TMA of queries and keys, warp 1 issues P V, warp 2 S (and has allocated TMEM), warp 3 TMA of values, then the sides' warps, then the summing warps.
#pragma once
#include "dn_attn_tc.cuh"

namespace dn {

constexpr int AP_MAX_BLOCKS = 1024;                    // row blocks of a launch at most
constexpr int AP_MAX_SORT = 256;                       // ... whose items may be dealt out whole
constexpr int AP_PART = 130 * 128;                     // floats of a partial output: [128 dims][128 rows], references, sums
constexpr int AP_OPITCH = HD + 16;                     // bytes of half a staged output row
constexpr int AP_SMEM = 5 * AT_TILE + 256 * AP_OPITCH + 3 * 2 * 2 * 128 * 4 + (AP_MAX_BLOCKS + 4) * 4 + (AP_MAX_BLOCKS + AP_MAX_SORT) * 2 + 256 + 1024;
constexpr int AP_MIN_RUN = 4;                          // places of a run at least, where items are cut
constexpr int AP_JOIN = 6;                             // places that the joining of cut items costs
constexpr int AP_HEAD = 1;                             // places of the line that an item has ahead of its tiles: what its end costs
template <int PARTS> struct ApShape {
  static constexpr int SIDES = PARTS == 2 ? 3 : 2, REGION = PARTS == 2 ? 128 : 192, SUM_WARPS = 8, WARPS = 4 + 4 * SIDES + SUM_WARPS, THREADS = 32 * WARPS;
  // setmaxnreg: of the 80 (96) a thread that 768 (640) threads are launched with
  static constexpr int LAUNCH = PARTS == 2 ? 80 : 96, R_UTIL = 40, R_SOFTMAX = PARTS == 2 ? 72 : 104, R_SUM = 112;
  static_assert(128 * R_UTIL + 128 * SIDES * R_SOFTMAX + 32 * SUM_WARPS * R_SUM <= THREADS * LAUNCH, "setmaxnreg split exceeds the CTA's launch allocation");
};

struct ApParams {
  bf16* out;                     // [tokens][n_heads][128]
  int n_heads, n_kv, G, TB;
  float scale;                   // of the scores, times log2(e)
  float* part;                   // [CTAs][2][AP_PART]
  unsigned int* count;           // [items], zero between launches
  unsigned int* err;
};
// one row block of an item: query rows [row0, + nq) at positions p_first .., pages [page0, pages) of its sequence
struct ApBlock { int row0, nq, p_first, page0, pages; const int32_t* bt; };

// The llama family's pages [page][K|V][kv head][64][128], one sequence, causal
struct ApPaged {
  const int32_t* block_table;
  const StepState* st;
  int T, n_kv, pos;
  static constexpr bool RISING = true;      // a row block has as many tiles as the one before or more
  __device__ __forceinline__ void start() { pos = st->pos; }
  __device__ __forceinline__ int blocks(int TB) const { return (T + TB - 1) / TB; }
  __device__ __forceinline__ ApBlock block(int b, int TB) const {
    ApBlock r;
    r.row0 = b * TB; r.nq = min(TB, T - b * TB); r.p_first = pos + b * TB; r.page0 = 0; r.pages = (r.p_first + r.nq + PAGE - 1) / PAGE; r.bt = block_table;
    return r;
  }
  __device__ __forceinline__ int lo(int) const { return 0; }      // first key position that a query sees
  __device__ __forceinline__ void at(int page, int kvh, int v, int half, int& c0, int& c1) const { c0 = half * 64; c1 = ((page * 2 + v) * n_kv + kvh) * PAGE; }
};

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
               ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}
__device__ __forceinline__ void tma_prefetch_map(const CUtensorMap* map) { asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory"); }
// mbar_wait for the two threads that issue products: asks again at once instead of sleeping until the barrier wakes it
__device__ __forceinline__ void mbar_spin(uint64_t* bar, uint32_t parity, unsigned int* err) {
  unsigned long long t0 = 0;
  for (unsigned it = 1;; ++it) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    if (ok) return;
    if ((it & 4095u) == 0) {
      const unsigned long long now = gtimer();
      if (t0 == 0) t0 = now;
      else if (now - t0 > MK_TIMEOUT_NS) { atomicExch(err, 2u); return; }
    }
  }
}
// from FROM registers a thread to TO, by a whole warpgroup (the direction has to be the right one)
template <int FROM, int TO>
__device__ __forceinline__ void ap_regs() {
  if constexpr (TO > FROM) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(TO));
  else if constexpr (TO < FROM) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(TO));
}
// 2^(a - b) of whole numbers a <= b (a may be -inf: 0)
__device__ __forceinline__ float ap_pow(float a, float b) { return a - b < -126.f || a == -INFINITY ? 0.f : __uint_as_float((uint32_t)(127 + (int)(a - b)) << 23); }

// the queries [tokens][heads][128] in boxes of 64 dims x a key head's `group` query heads x as many tokens as 128 rows hold (encode: cuTensorMapEncodeTiled)
template <class Encode>
inline bool query_map(Encode encode, CUtensorMap* out, const void* base, int tokens, int heads, int group) {
  if (!encode || !base) return false;
  cuuint64_t dims[3] = {128, (cuuint64_t)heads, (cuuint64_t)tokens};
  cuuint64_t strides[2] = {256, (cuuint64_t)heads * 256};
  cuuint32_t box[3] = {64, (cuuint32_t)group, (cuuint32_t)(128 / group)};
  cuuint32_t estr[3] = {1, 1, 1};
  return encode(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Items from which a launch takes this kernel; fewer stay with k_attn_prefill_tc, whose clusters share a row block's keys.  By the tokens alone, so that a chunk that
// is captured and replayed at other positions takes the kernel of an eager one.  With eight key heads of groups of 4, 200 tokens (56 items) behind 0 / 1,000 / 3,000 / 8,000:
// 12.4, 24.4, 35.2, 64 us there and 14.5, 31, 39, 61 here; 300 (80 items) 14.6, 26.8, 49, 104 and 15.5, 26.8, 45, 74.  Three parts: groups of 5, 100 tokens (32 items)
// behind 3,000 / 8,000 33, 53 and 38, 55; 150 (48) 43, 79 and 41, 62.
static inline bool attn_prompt_from(int G, int T, int n_kv) {
  const int TB = 128 / G, blocks = (T + TB - 1) / TB;
  return blocks <= AP_MAX_BLOCKS && n_kv * blocks >= (attn_parts(G, T) == 3 ? 40 : 72);
}

template <class Geom, int PARTS>
__global__ void __launch_bounds__(ApShape<PARTS>::THREADS, 1) k_attn_prompt(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapK,
                                                                           const __grid_constant__ CUtensorMap mapV, const ApParams p, const Geom geom_) {
  using Sh = ApShape<PARTS>;
  constexpr int SIDES = Sh::SIDES, REGION = Sh::REGION;
  extern __shared__ __align__(1024) unsigned char tc_smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char *sQ = smem, *sK = smem + AT_TILE, *sV = smem + 3 * AT_TILE;      // K, V: two buffers
  unsigned char* sO = smem + 5 * AT_TILE;                                        // [8 warps][32 rows][AP_OPITCH]
  float* info = reinterpret_cast<float*>(sO + 256 * AP_OPITCH);                  // [side][2][references, sums][128]
  int* pre = reinterpret_cast<int*>(info + 3 * 2 * 2 * 128);                     // places of the row blocks before each
  uint16_t* order = reinterpret_cast<uint16_t*>(pre + AP_MAX_BLOCKS + 2);        // row blocks, the longest first
  uint16_t* len = order + AP_MAX_SORT;                                           // places of a row block
  uint64_t* bars = reinterpret_cast<uint64_t*>(len + AP_MAX_BLOCKS);
  uint64_t *q_full = bars, *q_empty = bars + 1, *k_full = bars + 2, *k_empty = bars + 4, *v_full = bars + 6, *v_empty = bars + 9, *s_full = bars + 12, *p_full = bars + 15,
           *i_full = bars + 18, *o_full = bars + 24, *o_free = bars + 25, *r_free = bars + 26;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 29);
  int* last_s = reinterpret_cast<int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    mbar_init(q_full, 1); mbar_init(q_empty, 1); mbar_init(o_full, 1); mbar_init(o_free, Sh::SUM_WARPS);
    for (int i = 0; i < 2; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); }
    for (int i = 0; i < 3; ++i) { mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 4); mbar_init(&r_free[i], 1); }
    for (int i = 0; i < 6; ++i) mbar_init(&i_full[i], 4);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (threadIdx.x == 32) {
    tma_prefetch_map(&mapQ);
    tma_prefetch_map(&mapK);
    tma_prefetch_map(&mapV);
  }
  pdl_wait();
  Geom geom = geom_;
  geom.start();
  const int TB = p.TB, G = p.G, nb = geom.blocks(TB);
  const int items = p.n_kv * nb, ctas = (int)gridDim.x;
  const bool sortable = Geom::RISING || nb <= AP_MAX_SORT;
  for (int b = threadIdx.x; b < nb; b += Sh::THREADS) {
    const ApBlock k = geom.block(b, TB);
    len[b] = (uint16_t)((k.pages - k.page0 + 1) / 2 + AP_HEAD);
  }
  if (threadIdx.x == 0) pre[AP_MAX_BLOCKS + 1] = 0;
  __syncthreads();
  if (!Geom::RISING && sortable) {
    for (int b = threadIdx.x; b < nb; b += Sh::THREADS) {
      const int n = len[b];
      int place = 0;
      for (int x = 0; x < nb; ++x) place += len[x] > n || (len[x] == n && x > b);
      order[place] = (uint16_t)b;
    }
    __syncthreads();
  }
  // whole items: the i-th longest goes to CTA i, the next ones from the last CTA back to the first, and so on
  auto dealt = [&](int c, int k) { return k * ctas + ((k & 1) ? ctas - 1 - c : c); };
  auto block_of = [&](int i) { const int k = i / p.n_kv; return Geom::RISING ? nb - 1 - k : (int)order[k]; };
  if (warp == 0) {
    int sum = 0;
    for (int b = 0; b < nb; b += 32) {
      int s = b + lane < nb ? len[b + lane] : 0;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) { const int x = __shfl_up_sync(0xffffffffu, s, d); if (lane >= d) s += x; }
      if (b + lane < nb) pre[b + lane + 1] = sum + s;
      sum += __shfl_sync(0xffffffffu, s, 31);
    }
    if (lane == 0) pre[0] = 0;
  } else if (sortable) {
    int most = 0;
    for (int c = (int)threadIdx.x - 32; c < ctas; c += Sh::THREADS - 32) {
      int load = 0;
      for (int k = 0, i; (i = dealt(c, k)) < items; ++k) load += len[block_of(i)];
      most = max(most, load);
    }
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 0 && most) atomicMax(&pre[AP_MAX_BLOCKS + 1], most);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot, tO = tmem + 384;

  // this CTA's share: whole items, or an equal run of the line of all items' places, whichever is expected to take less
  const int P = pre[nb], total = p.n_kv * P, per = max((total + ctas - 1) / ctas, AP_MIN_RUN);
  const bool whole = sortable && pre[AP_MAX_BLOCKS + 1] <= per + AP_JOIN;
  const int u0 = min(total, (int)blockIdx.x * per), u1 = min(total, u0 + per);
  // the items of the share, one after the other: n tiles from the item's tile j0 on (none, where a run ends ahead of the item's first tile)
  struct Item { int u, h, b, j0, n; };      // u: whole items: how many came before; a run: its first place here
  auto enter = [&](Item& it, int r) {      // r: places of the item ahead of the run
    const int end = whole ? pre[it.b + 1] - pre[it.b] : min(pre[it.b + 1] - pre[it.b], u1 - (it.h * P + pre[it.b]));
    it.j0 = max(r - AP_HEAD, 0);
    it.n = max(end - AP_HEAD - it.j0, 0);
  };
  auto begin = [&](Item& it) {
    if (whole) {
      it.u = 0;
      const int i = min((int)blockIdx.x, items - 1);
      it.b = block_of(i);
      it.h = i % p.n_kv;
      enter(it, 0);
      return;
    }
    it.u = u0;
    it.h = u0 / P;
    const int r = u0 - it.h * P;
    int lo = 0, hi = nb;      // pre[lo] <= r < pre[hi]
    while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (pre[mid] <= r) lo = mid; else hi = mid; }
    it.b = lo;
    enter(it, r - pre[lo]);
  };
  auto more = [&](const Item& it) { return whole ? dealt((int)blockIdx.x, it.u) < items : it.u < u1; };
  auto next = [&](Item& it) {      // (what lies behind the share's end is not looked at)
    if (whole) {
      const int i = min(dealt((int)blockIdx.x, ++it.u), items - 1);
      it.b = block_of(i);
      it.h = i % p.n_kv;
    } else {
      if (++it.b == nb) { it.b = 0; ++it.h; }
      it.u = it.h * P + pre[it.b];
    }
    enter(it, 0);
  };

  if (warp < 4) {
    ap_regs<Sh::LAUNCH, Sh::R_UTIL>();
    if (warp == 0 || warp == 3) {
      // ===================== TMA: queries and keys; values =====================
      int g = 0, i = 0;
      Item it;
      for (begin(it); more(it); next(it)) {
        if (it.n == 0) continue;
        const ApBlock k = geom.block(it.b, TB);
        if (warp == 0 && lane == 0) {
          mbar_wait(q_empty, (uint32_t)(i & 1) ^ 1u, p.err);
          mbar_arrive_expect_tx(q_full, (uint32_t)(G * TB * 256));
          tma_load_3d(sQ, &mapQ, 0, it.h * G, k.row0, q_full);
          tma_load_3d(sQ + 16384, &mapQ, 64, it.h * G, k.row0, q_full);
        }
        ++i;
        int ids = 0;
        for (int j = 0; j < it.n; ++j, ++g) {
          if ((j & 15) == 0) ids = k.bt[min(k.page0 + 2 * (it.j0 + j) + lane, k.pages - 1)];      // (an unused half: any page of the sequence, masked)
          const int pg0 = __shfl_sync(0xffffffffu, ids, 2 * (j & 15)), pg1 = __shfl_sync(0xffffffffu, ids, 2 * (j & 15) + 1);
          if (lane != 0) continue;
          const int v = warp == 3, st = g & 1;
          uint64_t *full = v ? &v_full[st] : &k_full[st], *empty = v ? &v_empty[st] : &k_empty[st];
          unsigned char* dst = (v ? sV : sK) + st * AT_TILE;
          const CUtensorMap* map = v ? &mapV : &mapK;
          mbar_wait(empty, ((uint32_t)(g >> 1) & 1u) ^ 1u, p.err);
          mbar_arrive_expect_tx(full, AT_TILE);
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            int c0, c1, d0, d1;
            geom.at(pg0, it.h, v, hf, c0, c1);
            geom.at(pg1, it.h, v, hf, d0, d1);
            tma_load_2d(dst + hf * 16384, map, c0, c1, full);
            tma_load_2d(dst + hf * 16384 + 8192, map, d0, d1, full);
          }
        }
        __syncwarp();
      }
    } else if (warp == 2 && lane == 0) {
      // ===================== S.  (Two threads issue the two kinds of product, so that the waits of one fall into the other's products) =====================
      const uint32_t idesc = tc_instr_desc(128, 128);
      int g = 0, i = 0;
      Item it;
      for (begin(it); more(it); next(it)) {
        if (it.n == 0) continue;
        mbar_spin(q_full, (uint32_t)i++ & 1u, p.err);
        for (int j = 0; j < it.n; ++j, ++g) {
          const int st = g & 1, sd = g % SIDES;
          mbar_spin(&k_full[st], (uint32_t)(g >> 1) & 1u, p.err);
          mbar_spin(&r_free[sd], ((uint32_t)(g / SIDES) & 1u) ^ 1u, p.err);      // the product that read this region's weights is done
          tc_fence_after();
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint64_t adesc = tc_smem_desc(sQ + h * 16384), bdesc = tc_smem_desc(sK + st * AT_TILE + h * 16384);
#pragma unroll
            for (int k = 0; k < 4; ++k) tc_mma(tmem + sd * REGION, adesc + (uint64_t)(2 * k), bdesc + (uint64_t)(2 * k), idesc, (h | k) ? 1u : 0u);
          }
          tc_commit(&s_full[sd]);
          tc_commit(&k_empty[st]);
        }
        tc_commit(q_empty);
      }
    } else if (warp == 1 && lane == 0) {
      // ===================== P V =====================
      const uint32_t idesc = tc_instr_desc(128, 128) | (1u << 16);       // V is MN-major
      int tiles = 0;
      Item it;
      for (begin(it); more(it); next(it)) tiles += it.n;
      for (int g = 0; g < tiles; ++g) {
        const int st = g & 1, sd = g % SIDES;
        mbar_spin(&v_full[st], (uint32_t)(g >> 1) & 1u, p.err);
        mbar_spin(&p_full[sd], (uint32_t)(g / SIDES) & 1u, p.err);
        mbar_spin(o_free, ((uint32_t)g & 1u) ^ 1u, p.err);      // the product before has been read
        tc_fence_after();
        const uint64_t vdesc = tc_smem_desc_mn(sV + st * AT_TILE, 16384, 1024);
        const uint32_t tP = tmem + sd * REGION;
#pragma unroll
        for (int part = PARTS - 1; part >= 0; --part)      // the small parts first: fewer sums are cut at the size of the result
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            tc_mma_ts(tO, part == 2 ? tP + 128 + 8 * kk : tP + 16 * kk + 8 * part, vdesc + (uint64_t)(kk * (2048 >> 4)), idesc,
                      (part < PARTS - 1 || kk) ? 1u : 0u);
        tc_commit(o_full);
        tc_commit(&r_free[sd]);
        tc_commit(&v_empty[st]);
      }
    }
    __syncwarp();
  } else if (warp < 4 + 4 * SIDES) {
    // ===================== weights =====================
    ap_regs<Sh::LAUNCH, Sh::R_SOFTMAX>();
    const int sd = (warp - 4) >> 2, qd = warp & 3, r = qd * 32 + lane, t = r / G;      // side, TMEM lane quarter, this thread's row and its token
    const uint32_t tS = tmem + sd * REGION + ((uint32_t)(qd * 32) << 16);
    const float sc2 = p.scale;
    int g = 0;
    Item it;
    for (begin(it); more(it); g += it.n, next(it)) {
      const ApBlock k = geom.block(it.b, TB);
      const bool ok = t < k.nq && r < G * TB;
      const int pos = k.p_first + t, last = ok ? pos : -1, lo = ok ? geom.lo(pos) : 0, kv_max = k.p_first + k.nq;
      for (int j = (sd + SIDES - g % SIDES) % SIDES; j < it.n; j += SIDES) {
        const int gt = g + j, key0 = k.page0 * PAGE + ((it.j0 + j) << 7), nth = gt / SIDES;
        // every key of the tile is seen by every live row of the warp (rows without a query compute something that is not stored)
        const bool all_seen = __all_sync(0xffffffffu, !ok || (key0 + 127 <= pos && key0 >= lo));
        mbar_wait(&s_full[sd], (uint32_t)nth & 1u, p.err);
        __syncwarp();
        tc_fence_after();
        // (loops of few instructions: five warps a scheduler in three roles meet in its instruction cache)
        if (!all_seen) {      // scores of keys that the row does not see: -inf
#pragma unroll 1
          for (int c = 0; c < 128; c += 32) {
            uint32_t v[32];
            tm_ld32(tS + c, v);
            tm_wait_ld();
            tm_pin(v);
            const int first = lo - key0 - c, end = last - key0 - c;      // columns first .. end are seen
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (i > end || i < first) v[i] = 0xff800000u;
            tmem_st32(tS + c, v);
          }
          tm_wait_st();
        }
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll 1
        for (int c = 0; c < 128; c += 32) {
          uint32_t v[32];
          tm_ld32(tS + c, v);
          tm_wait_ld();
          tm_pin(v);
#pragma unroll
          for (int i = 0; i < 16; ++i) mx[i & 3] = fmaxf(fmaxf(mx[i & 3], __uint_as_float(v[i])), __uint_as_float(v[i + 16]));      // (one instruction)
        }
        const float ref = ceilf(fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * sc2);
        const float nref = ref == -INFINITY ? 0.f : -ref;
        float2 l0 = f2_of(0.f), l1 = l0;
        uint32_t va[2][16];
        tm_ld16(tS, va[0]);
#pragma unroll 1
        for (int c = 0; c < 128; c += 32)
#pragma unroll
          for (int z = 0; z < 2; ++z) {
            uint32_t (&v)[16] = va[z], hi[8], lo[8], x[8];
            tm_wait_ld();
            tm_pin16(v);
            if (z == 0 || c < 96) tm_ld16(tS + c + 16 * z + 16, va[z ^ 1]);      // on its way while this one's weights are formed
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float2 y = f2_fma(f2_bits(v[2 * i], v[2 * i + 1]), f2_of(sc2), f2_of(nref));
              float2 e = make_float2(tc_ex2(y.x), tc_ex2(y.y));
              if (i & 1) l1 = f2_add(l1, e); else l0 = f2_add(l0, e);
              if (PARTS == 3) {      // cut, not rounded: three times eight bits hold all 24
                hi[i] = upper_halves(e.x, e.y);
                e = below_upper_halves(e);
                lo[i] = upper_halves(e.x, e.y);
                e = below_upper_halves(e);
                x[i] = upper_halves(e.x, e.y);
              } else {
                hi[i] = pack_bf16x2(e.x, e.y);
                e = f2_fma(f2_bits(hi[i] << 16, hi[i] & 0xffff0000u), f2_of(-1.f), e);
                lo[i] = pack_bf16x2(e.x, e.y);
              }
            }
            tm_st8(tS + c + 16 * z, hi);
            tm_st8(tS + c + 16 * z + 8, lo);
            if constexpr (PARTS == 3) tm_st8(tS + 128 + c / 2 + 8 * z, x);
          }
        l0 = f2_add(l0, l1);
        float* in = info + (sd * 2 + (nth & 1)) * 256 + r;
        in[0] = ref;
        in[128] = l0.x + l0.y;
        if (key0 + 128 > kv_max) {      // value rows that belong to no key: whatever the page holds, it must not enter
          const int valid = kv_max - key0;
          unsigned char* vt = sV + (gt & 1) * AT_TILE;
          mbar_wait(&v_full[gt & 1], (uint32_t)(gt >> 1) & 1u, p.err);
          for (int i = (int)threadIdx.x - 128 - sd * 128; i < (128 - valid) * 16; i += 128) {
            const int row = valid + (i >> 4), c = i & 15;
            *reinterpret_cast<uint4*>(vt + (c >> 3) * 16384 + row * 128 + (c & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        tm_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) { mbar_arrive(&p_full[sd]); mbar_arrive(&i_full[sd * 2 + (nth & 1)]); }
      }
    }
  } else {
    // ===================== sums and output =====================
    ap_regs<Sh::LAUNCH, Sh::R_SUM>();
    const int qd = warp & 3, hf = (warp - 4 - 4 * SIDES) >> 2, r = qd * 32 + lane;      // (two threads a row, half of the dims each)
    const uint32_t tOl = tO + hf * 64 + ((uint32_t)(qd * 32) << 16);
    int g = 0;
    Item it, cut[2];      // the items that the run's ends cut: parts of them are left to be joined
    int n_cut = 0;
    const int over_g = 65536 / G + 1;      // row / G of rows below 128
    unsigned char* mine_s = sO + (warp - 4 - 4 * SIDES) * 32 * AP_OPITCH;      // this warp's 32 rows of 64 dims
    auto put = [&](const Item& x, const float2 (&o)[32], float L) {      // the item's output, by way of shared memory: whole lines of four rows a store
      const ApBlock k = geom.block(x.b, TB);
      const float inv = 1.0f / L;
      __syncwarp();
#pragma unroll
      for (int c = 0; c < 8; ++c)
        *reinterpret_cast<uint4*>(mine_s + lane * AP_OPITCH + c * 16) =
            make_uint4(pack_bf16x2(o[4 * c].x * inv, o[4 * c].y * inv), pack_bf16x2(o[4 * c + 1].x * inv, o[4 * c + 1].y * inv),
                       pack_bf16x2(o[4 * c + 2].x * inv, o[4 * c + 2].y * inv), pack_bf16x2(o[4 * c + 3].x * inv, o[4 * c + 3].y * inv));
      __syncwarp();
      const int limit = min(G * k.nq, G * TB);      // rows with a query
      bf16* dst = p.out + ((size_t)k.row0 * p.n_heads + x.h * G) * HD + hf * 64 + (lane & 7) * 8;
#pragma unroll 1
      for (int i = 0; i < 8; ++i) {
        const int rr = i * 4 + (lane >> 3), row = qd * 32 + rr, tt = (row * over_g) >> 16;
        if (row < limit) *reinterpret_cast<uint4*>(dst + ((size_t)tt * p.n_heads + row - tt * G) * HD) = *reinterpret_cast<const uint4*>(mine_s + rr * AP_OPITCH + (lane & 7) * 16);
      }
    };
    auto item_tiles = [&](const Item& x) { return pre[x.b + 1] - pre[x.b] - AP_HEAD; };
    float M = -INFINITY, L = 0.f;
    float2 o[32];
    for (begin(it); more(it); next(it)) {
      if (it.n == 0) continue;
      M = -INFINITY;
      L = 0.f;
#pragma unroll
      for (int i = 0; i < 32; ++i) o[i] = f2_of(0.f);
#pragma unroll 1
      for (int j = 0; j < it.n; ++j, ++g) {
        const int sd = g % SIDES, nth = g / SIDES;
        mbar_wait(&i_full[sd * 2 + (nth & 1)], (uint32_t)(nth >> 1) & 1u, p.err);
        const float* in = info + (sd * 2 + (nth & 1)) * 256 + r;
        const float ref = in[0], top = fmaxf(M, ref), a = ap_pow(M, top), b = ap_pow(ref, top);
        M = top;
        L = fmaf(L, a, in[128] * b);
        mbar_wait(o_full, (uint32_t)g & 1u, p.err);
        __syncwarp();
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t v[32];
          tm_ld32(tOl + c * 32, v);
          tm_wait_ld();
          tm_pin(v);
          if (c == 1) {      // the next product may come
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(o_free);
          }
#pragma unroll
          for (int i = 0; i < 16; ++i) o[c * 16 + i] = f2_fma(o[c * 16 + i], f2_of(a), f2_mul(f2_bits(v[2 * i], v[2 * i + 1]), f2_of(b)));
        }
      }
      if (it.n < item_tiles(it)) {
        float* mine = p.part + ((size_t)blockIdx.x * 2 + (it.j0 == 0)) * AP_PART + r;
#pragma unroll
        for (int i = 0; i < 32; ++i) { __stcg(mine + (hf * 64 + 2 * i) * 128, o[i].x); __stcg(mine + (hf * 64 + 2 * i + 1) * 128, o[i].y); }
        if (hf == 0) { __stcg(mine + 128 * 128, M); __stcg(mine + 129 * 128, L); }
        cut[it.j0 == 0] = it;
        n_cut |= it.j0 == 0 ? 2 : 1;
      } else put(it, o, L);
    }
    if (n_cut) {
      __threadfence();
      asm volatile("bar.sync 1, %0;" ::"n"(32 * Sh::SUM_WARPS) : "memory");
      auto first_of = [&](const Item& x) { return (x.h * P + pre[x.b] + AP_HEAD) / per; };
      auto pieces_of = [&](const Item& x) { return (x.h * P + pre[x.b + 1] - 1) / per - first_of(x) + 1; };
      if (qd == 0 && hf == 0 && lane < 2) {
        bool last = false;
        if (n_cut >> lane & 1) {
          const Item& x = cut[lane];
          unsigned int* c = p.count + x.h * nb + x.b;
          last = atomicAdd(c, 1u) == (unsigned)(pieces_of(x) - 1);
          if (last) *c = 0u;
        }
        last_s[lane] = last;
      }
      asm volatile("bar.sync 1, %0;" ::"n"(32 * Sh::SUM_WARPS) : "memory");
      __threadfence();
#pragma unroll 1
      for (int x = 1; x >= 0; --x) {      // (the item that the run's end cuts first: its first piece is still in registers)
        if (!last_s[x]) continue;
        const Item w = x ? cut[1] : cut[0];
        const int first = first_of(w), pieces = pieces_of(w);
        if (x == 0) {
          M = -INFINITY;
          L = 0.f;
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = f2_of(0.f);
        }
#pragma unroll 1
        for (int z = x; z < pieces; ++z) {      // the first piece is its CTA's last one, the others are their CTAs' first
          const float* q = p.part + ((size_t)(first + z) * 2 + (z == 0)) * AP_PART + r;
          const float ref = __ldcg(q + 128 * 128), top = fmaxf(M, ref), a = ap_pow(M, top), b = ap_pow(ref, top);
          M = top;
          L = fmaf(L, a, __ldcg(q + 129 * 128) * b);
#pragma unroll
          for (int i = 0; i < 32; ++i)
            o[i] = f2_fma(o[i], f2_of(a), f2_mul(make_float2(__ldcg(q + (hf * 64 + 2 * i) * 128), __ldcg(q + (hf * 64 + 2 * i + 1) * 128)), f2_of(b)));
        }
        put(w, o, L);
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
