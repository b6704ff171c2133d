// dn_seq_delta_chunk.cuh -- the gated delta rule of prompt portions, 32 tokens at a time (libdnet_b200_seq.so, bf16 models).
//
// k_delta_rule takes a token after the other: S <- g S; u = beta (v - S^T k); S <- S + k u^T; o = S^T q.  Within a chunk that starts from S0, with
// G_t = g_1 .. g_t and D_ts = g_(s+1) .. g_t (s <= t), the same numbers are
//     (I + L) U = beta (V - G K S0)      L_ts = beta_t D_ts (k_t . k_s), s < t      (a row a token)
//     O = G Q S0 + A U                   A_ts = D_ts (q_t . k_s), s <= t
//     S = G_32 S0 + K^T (D_32 U)
// so that only three products of 32 tokens with S are left in the serial chain.  k_delta_chunk_prep forms, for all chunks at once, what does not
// depend on S: T = (I + L)^-1 beta by forward substitution (its rows are those of a product of contractions: no entry is above 1) and A, in fp32.
// k_delta_chunk walks the chunks of one (entry, head), four warps with 16 columns of S each, transposed in the accumulators' layout: S^T, V^T - .. and U^T
// are the A operands of mma.sync straight from the registers that hold them, K, Q, T and A come as B operands from shared memory (one bulk copy each, one
// chunk ahead).
//
// fp32 on 16-bit matrix instructions: every operand is three parts of bf16, all 24 bits, and six of the nine products are formed (the others are below
// 2^-25); the sums of sixteen products of the large parts meet in fp32 additions, the small ones in an accumulator of their own, and the state's products, 32 deep, in one
// chain, the small ones first: what is added to the state is then rounded once.  T's diagonal, beta, is not part of the product, products of decays are formed in 64 bits and
// rounded once, A not before it is in parts, and never as quotients: a decay of 0 is as good as any.  Error against 64 bits (2-norm, 1e-8), outputs / states, and token by token:
//   decays of about 0.8, entries of 81 to 250 tokens, 8 heads of 128 x 128 6.3 / 5.7, 7.1 / 6.3; 64 x 96, 95 and 130 tokens 6.5 / 5.7, 7.3 / 6.0; 1,500 tokens 6.1 / 5.4, 6.7 / 6.8
//   decays near 1 and keys that are nearly alike, 1,500 tokens 23 / 29, 89 / 122; decays of 0, 1e-20 and 1 5.1 / 4.0, 6.4 / 4.5
// (Two parts of fp16 and three products are a third faster and three times further off.  tests/test_gpu_delta_chunks.py holds these.)
//
// Bound by mma.sync, 348 a chunk and warp at 8.7 cycles each, and the splitting into parts beside them, which one warp a scheduler does not hide.  32 heads of
// 128 x 128, microseconds, token by token / preparation + chunks: four entries, 2,048 tokens, the longest 788: 450 / 27 + 175; one entry of 2,048: 630 / 27 + 246; one of
// 100: 36 / 12.6 + 20; one of 16: 10.5 / 11 + 8.5.
#pragma once
#include "dn_seq_kernels.cuh"
#include "dn_megakernel.cuh"

namespace dnseq {

constexpr int DC = 32;                          // tokens of a chunk
// Entries from this many tokens on; shorter ones stay with k_delta_rule (a chunk takes as long however few of its tokens there are, and the preparation 11 us).
// Token by token / preparation + chunks, microseconds, entries x heads of 128 x 128 (64 x 64): one entry of 8 heads, 80 tokens 29 / 29 (25 / 23), 96 35 / 29 (29 / 24), 128 45 / 33
// (37 / 27); 96 in all, 80 tokens 46 / 50 (29 / 27), 96 54 / 50 (33 / 27), 112 62 / 60; 192, 80 tokens 82 / 68 (33 / 38), 112 111 / 85 (45 / 49), 128 124 / 87 (50 / 50); 512, 80 tokens
// 168 / 150 (62 / 71), 112 229 / 190 (83 / 91), 128 259 / 191 (94 / 93), 160 319 / 230 (115 / 111).  From these lines on chunks are slower nowhere, but for 5 % with keys of 64
// and 512 in all whose last chunk is half empty (144 tokens 105 / 109).
constexpr int DC_FROM = 96, DC_FROM_64 = 128;      // (of keys of 128 and of 64)
__host__ __device__ __forceinline__ int dc_from(int dk) { return dk == 64 ? DC_FROM_64 : DC_FROM; }
__host__ __device__ __forceinline__ int dc_chunks(int tokens, int dk) { return tokens >= dc_from(dk) ? (tokens + DC - 1) / DC : 0; }
constexpr int DC_TP = DC + 8;                   // row pitch of T and A, of K and Q dk + 8: eight rows of 16 bytes fall into different banks
__host__ __device__ constexpr int dc_k_bytes(int dk) { return 3 * DC * (dk + 8) * 2; }       // [3 parts][32][dk + 8] bf16 of a (chunk, key head): K, then as many of Q
constexpr int DC_TA_NUMBERS = 6 * DC * DC_TP;                                                // [T, A][3 parts][32][40] bf16 of a (chunk, head),
constexpr int DC_TA_BYTES = DC_TA_NUMBERS * 2 + 3 * DC * 4;                                  // then G_t, D_32,s and beta_t [32] in fp32
constexpr int DC_XCH = 24;                      // numbers that a thread hands to the other half's
// shared memory: K of two chunks, Q, T and A, V [32][16 cg + 4], what the halves exchange
__host__ __device__ constexpr size_t dc_smem(int dk, int cg) { return (size_t)3 * dc_k_bytes(dk) + DC_TA_BYTES + (DC * (16 * cg + 4) + 2 * cg * DC_XCH * 32) * 4 + 64; }
// K and Q in parts (later the L [32][36] of four heads); k_t . k_s and q_t . k_s; decays and betas of a warp's head
constexpr int DC_PREP_WARPS = 8;
__host__ __device__ constexpr size_t dc_prep_smem(int dk) { return (size_t)2 * dc_k_bytes(dk) + 2 * DC * (DC + 1) * 8 + DC_PREP_WARPS * 2 * DC * 4; }

// 64 columns a block (of one an SM) where the blocks of the entries that are cut nearly fill the SMs, else 32 (two an SM): a block of 64 reads K and Q half
// as often, one of 32 has a warp a scheduler to itself.  Four entries of 32 heads (256 blocks of 64), the longest 788: 175 us with 64, 210 with 32; two of 700 (128): 111, 120; of
// 16 heads (64): 113, 88; one entry of 2,048, 32 heads: 310, 246.
__host__ __device__ __forceinline__ bool dc_wide(int blocks, int sms) { return 4 * blocks >= 3 * sms; }

// two numbers (x + ex, y + ey, where ex and ey are below the last place) in three parts of bf16: all 24 bits
__device__ __forceinline__ void split3(float x, float y, uint32_t (&p)[3], float ex = 0.f, float ey = 0.f) {
#pragma unroll
  for (int i = 0; i < 3; i++) {
    if (i == 2) { x += ex; y += ey; }
    p[i] = pack_bf16(x, y);
    x -= __uint_as_float(p[i] << 16);
    y -= __uint_as_float(p[i] & 0xffff0000u);
  }
}
// The instruction cuts its sums to fp32 instead of rounding them, so that a product of the large parts is too small by some part of 2^-24 on average: K and Q are made
// larger by as much as measured best (outputs / states against 64 bits, 1e-8, decays of about 0.8, 1,500 tokens: 0 / 0 6.9 / 6.8, 0.35 / 0.35 6.3 / 5.7, 0.5 / 0.3 6.1 / 5.4,
// 0.7 / 0.5 8.2 / 5.2; token by token 6.7 / 6.8).
constexpr float DC_CUT_K = 0.5f / 16777216.f, DC_CUT_Q = 0.3f / 16777216.f;
__device__ __forceinline__ void dc_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void dc_mma0(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {      // from zero
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void add_pair(float& x, float& y, float a, float b) {      // two fp32 additions
  asm("{.reg .b64 u, v, w; mov.b64 u, {%0, %1}; mov.b64 v, {%2, %3}; add.rn.f32x2 w, u, v; mov.b64 {%0, %1}, w;}" : "+f"(x), "+f"(y) : "f"(a), "f"(b));
}
// sixteen products deep, NT tiles of eight columns: small gets the five products of parts that matter beside that of the large ones (the three left out are below 2^-25 of
// the result)
template <int NT>
__device__ __forceinline__ void mma_small(float (&small)[NT][4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][2 * NT]) {
#pragma unroll
  for (int n = 0; n < NT; n++) dc_mma(small[n], a[2], b[0][2 * n], b[0][2 * n + 1]);
#pragma unroll
  for (int n = 0; n < NT; n++) dc_mma(small[n], a[0], b[2][2 * n], b[2][2 * n + 1]);
#pragma unroll
  for (int n = 0; n < NT; n++) dc_mma(small[n], a[1], b[1][2 * n], b[1][2 * n + 1]);
#pragma unroll
  for (int n = 0; n < NT; n++) dc_mma(small[n], a[1], b[0][2 * n], b[0][2 * n + 1]);
#pragma unroll
  for (int n = 0; n < NT; n++) dc_mma(small[n], a[0], b[1][2 * n], b[1][2 * n + 1]);
}
// ... and c the sums of the large parts' products by fp32 additions
template <int NT>
__device__ __forceinline__ void mma_parts(float (&c)[NT][4], float (&small)[NT][4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][2 * NT]) {
  float d[NT][4];
#pragma unroll
  for (int n = 0; n < NT; n++) dc_mma0(d[n], a[0], b[0][2 * n], b[0][2 * n + 1]);
  mma_small(small, a, b);
#pragma unroll
  for (int n = 0; n < NT; n++) {
    add_pair(c[n][0], c[n][1], d[n][0], d[n][1]);
    add_pair(c[n][2], c[n][3], d[n][2], d[n][3]);
  }
}
template <int NT>
__device__ __forceinline__ void zero_tiles(float (&c)[NT][4]) {
#pragma unroll
  for (int n = 0; n < NT; n++) c[n][0] = c[n][1] = c[n][2] = c[n][3] = 0.f;
}
// A fragment (three parts) of sixteen reduction places from two accumulator tiles
__device__ __forceinline__ void a_frag(const float (&x)[4], const float (&y)[4], uint32_t (&a)[3][4]) {
  uint32_t p[3];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    if (i < 2) split3(x[2 * i], x[2 * i + 1], p); else split3(y[2 * i - 4], y[2 * i - 3], p);
    a[0][i] = p[0]; a[1][i] = p[1]; a[2][i] = p[2];
  }
}
// Numbers that are not finite.  The zeros above T's and A's diagonals meet the rows of later tokens, and 0 x NaN would carry such a number back to tokens before it: a column's
// rows from the first one on are taken as zeros, and its outputs from there on and its state become NaN, as token by token they are not finite from there on.  (Above bf16's largest,
// 3.39e38, is infinite here.)
constexpr float DC_LARGEST = 0x1.fep127f;
constexpr int DC_ALL_FINITE = DC | DC << 8;      // the first such token of a thread's two columns, a byte each; 32: none
// at(i): tokens 8 i + 2 (lane & 3) + {0, 1} of the first column ([0], [1]) and of the second
template <class At>
__device__ __forceinline__ int first_not_finite(At at, int lane, int before) {
  bool ok = true;
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) ok = ok && fabsf(at(i)[j]) <= DC_LARGEST;
  if (__all_sync(0xffffffffu, ok && before == DC_ALL_FINITE)) return before;
  int a = before & 255, b = before >> 8;
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int t = 8 * i + 2 * (lane & 3) + (j & 1);
      if (fabsf(at(i)[j]) <= DC_LARGEST) continue;
      if (j < 2) a = min(a, t); else b = min(b, t);
    }
#pragma unroll
  for (int d = 1; d < 4; d <<= 1) {
    a = min(a, __shfl_xor_sync(0xffffffffu, a, d));
    b = min(b, __shfl_xor_sync(0xffffffffu, b, d));
  }
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (8 * i + 2 * (lane & 3) + (j & 1) >= (j < 2 ? a : b)) at(i)[j] = 0.f;
  return a | b << 8;
}
// untiled copy into this CTA's shared memory; both addresses on 16 bytes, a multiple of 16 bytes
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dn::smem_u32(dst)), "l"(src), "r"(bytes), "r"(dn::smem_u32(bar)) : "memory");
}

// which entry a chunk belongs to, and which of its chunks it is (false: none)
__device__ __forceinline__ bool chunk_entry(const Batch& b, int dk, int chunk, int& e, int& c) {
  c = chunk;
  for (e = 0; e < b.E; e++) {
    const int nc = dc_chunks(b.ent_start[e + 1] - b.ent_start[e], dk);
    if (c < nc) return true;
    c -= nc;
  }
  return false;
}

// grid (chunks, key heads)
template <int DK>
__global__ void __launch_bounds__(32 * DC_PREP_WARPS) k_delta_chunk_prep(Batch b, int H, int G, const float* __restrict__ qn, const float* __restrict__ kn,
                                                                         const float* __restrict__ beta, const float* __restrict__ decay, bf16* __restrict__ kq,
                                                                         unsigned char* __restrict__ ta) {
  extern __shared__ __align__(128) unsigned char dcr[];
  constexpr int HP = DK + 8, LP = DC + 4;
  bf16* parts = reinterpret_cast<bf16*>(dcr);      // [K, Q][3][32][dk + 8]
  double *kk = reinterpret_cast<double*>(dcr + 2 * dc_k_bytes(DK)), *qk = kk + DC * (DC + 1);
  float* gb = reinterpret_cast<float*>(qk + DC * (DC + 1));
  static_assert(DC_PREP_WARPS / 2 * DC * LP * 4 <= 2 * dc_k_bytes(DK), "L lies over the parts");
  int e, c;
  if (!chunk_entry(b, DK, blockIdx.x, e, c)) return;
  const int g = blockIdx.y, n0 = b.ent_start[e] + c * DC, cnt = min(DC, b.ent_start[e + 1] - n0), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  bf16* out = kq + ((size_t)blockIdx.x * G + g) * dc_k_bytes(DK);      // (2 x dc_k_bytes bytes)
#pragma unroll 8
  for (int i = threadIdx.x; i < 2 * DC * (DK / 4); i += 32 * DC_PREP_WARPS) {
    const int z = i / (DC * (DK / 4)), t = i / (DK / 4) % DC, d = i % (DK / 4) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t < cnt) v = *reinterpret_cast<const float4*>((z ? qn : kn) + ((size_t)(n0 + t) * G + g) * DK + d);
    uint32_t p[3], q[3];
    const float more = z ? DC_CUT_Q : DC_CUT_K;
    split3(v.x, v.y, p, v.x * more, v.y * more);
    split3(v.z, v.w, q, v.z * more, v.w * more);
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const int at = ((3 * z + j) * DC + t) * HP + d;
      *reinterpret_cast<uint2*>(out + at) = *reinterpret_cast<uint2*>(parts + at) = make_uint2(p[j], q[j]);
    }
  }
  __syncthreads();
  // k_t . k_s (warps 0 .. 3) and q_t . k_s (4 .. 7), s <= t: sixteen tokens t and s a warp; the sums of sixteen products meet in 64 bits, for an error here
  // is the same for all columns of the state
  {
    const int z = warp >> 2, th = (warp >> 1) & 1, j = warp & 1;
    const bf16* A = parts + 3 * z * DC * HP;
    double sum[2][4];
#pragma unroll
    for (int n = 0; n < 2; n++) sum[n][0] = sum[n][1] = sum[n][2] = sum[n][3] = 0.;
    if (j <= th) {
#pragma unroll 2
      for (int k = 0; k < DK / 16; k++) {
        uint32_t a[3][4], f[3][4];
        float x[2][4], small[2][4];
        zero_tiles(x);
        zero_tiles(small);
#pragma unroll
        for (int p = 0; p < 3; p++) {
          ldsm_x4(a[p], A + (p * DC + th * 16 + (lane & 15)) * HP + k * 16 + (lane >> 4) * 8);
          ldsm_x4(f[p], parts + (p * DC + j * 16 + (lane >> 4) * 8 + (lane & 7)) * HP + k * 16 + ((lane >> 3) & 1) * 8);
        }
        mma_parts(x, small, a, f);
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
          for (int i = 0; i < 4; i++) sum[n][i] += (double)x[n][i] + (double)small[n][i];
      }
    }
    double* to = z ? qk : kk;
#pragma unroll
    for (int n = 0; n < 2; n++)
#pragma unroll
      for (int i = 0; i < 4; i++) to[(th * 16 + (lane >> 2) + (i & 2) * 4) * (DC + 1) + j * 16 + n * 8 + 2 * (lane & 3) + (i & 1)] = sum[n][i];
  }
  __syncthreads();
  // a head by two warps: T by the first, A and the decays by the second.  (The decays' products in 64 bits, rounded once: an error here is the same for all
  // numbers of a column and does not average out.)
  const int R = H / G, role = warp >> 2;
  float *L = reinterpret_cast<float*>(dcr) + (warp & 3) * DC * LP, *gs = gb + warp * 2 * DC, *bs = gs + DC;
  for (int r = warp & 3; r < R; r += 4) {
    const int h = g * R + r;
    const float gt = lane < cnt ? decay[(size_t)(n0 + lane) * H + h] : 1.f, bt = lane < cnt ? beta[(size_t)(n0 + lane) * H + h] : 0.f;
    __syncwarp();
    gs[lane] = gt;
    bs[lane] = bt;
    __syncwarp();
    unsigned char* base = ta + ((size_t)blockIdx.x * H + h) * DC_TA_BYTES;
    bf16* to = reinterpret_cast<bf16*>(base) + role * 3 * DC * DC_TP;
    auto store = [&](int t, auto x) {      // a number of T (fp32) or A (64 bits) in its parts
#pragma unroll
      for (int j = 0; j < 3; j++) {
        const bf16 v = __float2bfloat16_rn((float)x);
        to[(j * DC + t) * DC_TP + lane] = v;
        x -= __bfloat162float(v);
      }
    };
    double D = 0., Gt = 1.;      // D: of (t, s = lane)
    if (role) {
      float mine = 1.f;
#pragma unroll 4
      for (int t = 0; t < DC; t++) {
        const double gd = gs[t];
        D = lane == t ? 1. : D * gd;
        Gt *= gd;
        if (lane == t) mine = (float)Gt;
        store(t, lane <= t ? D * qk[t * (DC + 1) + lane] : 0.);
      }
      float* gm = reinterpret_cast<float*>(base + DC_TA_NUMBERS * 2);
      gm[lane] = mine;
      gm[DC + lane] = (float)D;
      continue;
    }
#pragma unroll 4
    for (int t = 0; t < DC; t++) {
      D = lane == t ? 1. : D * (double)gs[t];
      L[t * LP + lane] = lane < t ? (float)(D * kk[t * (DC + 1) + lane] * (double)bs[t]) : 0.f;
    }
    __syncwarp();
    float T[DC];      // column `lane` of the inverse
#pragma unroll
    for (int t = 0; t < DC; t++) {
      float a[4] = {lane == t ? 1.f : 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int s = 0; s < t; s += 4) {
        const float4 l = *reinterpret_cast<const float4*>(L + t * LP + s);
        a[0] = fmaf(-l.x, T[s], a[0]);
        if (s + 1 < t) a[1] = fmaf(-l.y, T[s + 1], a[1]);
        if (s + 2 < t) a[2] = fmaf(-l.z, T[s + 2], a[2]);
        if (s + 3 < t) a[3] = fmaf(-l.w, T[s + 3], a[3]);
      }
      T[t] = (a[0] + a[1]) + (a[2] + a[3]);
      store(t, lane < t ? T[t] * bt : 0.f);
    }
    reinterpret_cast<float*>(base + DC_TA_NUMBERS * 2)[2 * DC + lane] = bt;
  }
}

// grid (entries that are cut x heads, columns / (16 CG)), 64 CG threads: warp w has the columns of group w % CG and half of their rows (w / CG); the two halves' sums with K
// and Q meet in shared memory, and each finishes half of the tokens' outputs
template <int DK, int CG>
__global__ void __launch_bounds__(64 * CG, 4 / CG) k_delta_chunk(Batch b, int H, int G, int dv, const bf16* __restrict__ kq, const unsigned char* __restrict__ ta,
                                                                 const float* __restrict__ vv, float* __restrict__ state, size_t slot_stride, float* __restrict__ o,
                                                                 unsigned int* __restrict__ err) {
  extern __shared__ __align__(128) unsigned char dcr[];
  constexpr int HP = DK + 8, NT = DK / 16, KB = dc_k_bytes(DK), COLS = 16 * CG, VP = COLS + 4;
  unsigned char *sK = dcr, *sQ = dcr + 2 * KB, *sT = dcr + 3 * KB;
  const bf16* Ts = reinterpret_cast<const bf16*>(sT);
  const float *gm = reinterpret_cast<const float*>(sT + DC_TA_NUMBERS * 2), *Vs = gm + 3 * DC;
  float* xch = reinterpret_cast<float*>(sT + DC_TA_BYTES) + DC * VP;
  uint64_t *k_full = reinterpret_cast<uint64_t*>(xch + 2 * CG * DC_XCH * 32), *q_full = k_full + 2, *t_full = k_full + 3, *k_free = k_full + 4, *q_free = k_full + 5,
           *t_free = k_full + 6;      // (free: a warp each has read it out)
  __shared__ int pick;
  const int h = blockIdx.x % H, g = h / (H / G), lane = threadIdx.x & 31, warp = threadIdx.x >> 5, cg = warp % CG, hf = warp / CG;
  // the entry of this place in the order of lengths: the longest start first, and those that are not cut come last, behind the grid
  for (int i = threadIdx.x; i < b.E; i += blockDim.x) {
    const int n = b.ent_start[i + 1] - b.ent_start[i];
    int place = 0;
    for (int j = 0; j < b.E; j++) {
      const int m = b.ent_start[j + 1] - b.ent_start[j];
      place += m > n || (m == n && j < i);
    }
    if (place == (int)blockIdx.x / H) pick = i;
  }
  const int col0 = blockIdx.y * COLS, wide = min(COLS, dv - col0);      // columns of the block
  const int col = cg * 16 + (lane >> 2);      // this thread's columns of the block: col and col + 8
  const bool okA = col < wide, okB = col + 8 < wide;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 7; i++) dn::mbar_init(&k_full[i], i < 4 ? 1 : 2 * CG);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const int e = pick;
  int base = 0;      // chunks of the entries before this one
  for (int i = 0; i < e; i++) base += dc_chunks(b.ent_start[i + 1] - b.ent_start[i], DK);
  const int s0 = b.ent_start[e], len = b.ent_start[e + 1] - s0, chunks = dc_chunks(len, DK), Cv = H * dv;
  auto part = [&](unsigned char* dst, int c, int z, uint64_t* bar) {      // K (z = 0) or Q of chunk c
    if (lane == 0) {
      dn::mbar_arrive_expect_tx(bar, KB);
      bulk_copy(dst, reinterpret_cast<const unsigned char*>(kq) + ((size_t)(base + c) * G + g) * 2 * KB + z * KB, KB, bar);
    }
  };
  auto rest = [&](int c) {      // T, A and the values
    const int n0 = s0 + c * DC, cnt = min(DC, len - c * DC);
    if (lane == 0) {
      dn::mbar_arrive_expect_tx(t_full, DC_TA_BYTES + cnt * wide * 4);
      bulk_copy(sT, ta + ((size_t)(base + c) * H + h) * DC_TA_BYTES, DC_TA_BYTES, t_full);
    }
    __syncwarp();
    if (lane < cnt) bulk_copy(sT + DC_TA_BYTES + lane * VP * 4, vv + (size_t)(n0 + lane) * Cv + (size_t)h * dv + col0, wide * 4, t_full);
  };
  if (warp == 0) {
    part(sK, 0, 0, &k_full[0]);
    part(sQ, 0, 1, q_full);
    rest(0);
  }
  // S^T: tile i holds state rows hf dk / 2 + 8 i + 2 (lane & 3) + {0, 1} of column col ([0], [1]) and col + 8 ([2], [3])
  float* Sg = state + (size_t)b.ent_slot[e] * slot_stride + (size_t)h * DK * dv + (size_t)hf * (DK / 2) * dv + col0 + col;
  float S[NT][4];
#pragma unroll
  for (int i = 0; i < NT; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int d = 8 * i + 2 * (lane & 3) + (j & 1);
      S[i][j] = (j < 2 ? okA : okB) ? Sg[(size_t)d * dv + (j < 2 ? 0 : 8)] : 0.f;
    }
  const int brow = (lane >> 4) * 8 + (lane & 7), bcol = ((lane >> 3) & 1) * 8;      // ldmatrix: this lane's row of 16 tokens and first of 8 of the 16 numbers
  for (int c = 0; c < chunks; c++) {
    const bf16 *Ks = reinterpret_cast<const bf16*>(sK + (c & 1) * KB) + hf * (DK / 2), *Qs = reinterpret_cast<const bf16*>(sQ) + hf * (DK / 2);
    const int n0 = s0 + c * DC, cnt = min(DC, len - c * DC);
    // K S0 and Q S0, transposed
    float r[4][4], y[4][4], rs[4][4], ys[4][4];
    zero_tiles(r);
    zero_tiles(y);
    zero_tiles(rs);
    zero_tiles(ys);
    {
      dn::mbar_wait(&k_full[c & 1], (c >> 1) & 1, err);
      dn::mbar_wait(q_full, c & 1, err);
      __syncwarp();
#pragma unroll
      for (int k = 0; k < DK / 32; k++) {
        uint32_t a[3][4], f[3][8];
        a_frag(S[2 * k], S[2 * k + 1], a);
        auto load = [&](const bf16* src) {
#pragma unroll
          for (int p = 0; p < 3; p++)
#pragma unroll
            for (int j = 0; j < 2; j++) {
              uint32_t w[4];
              ldsm_x4(w, src + (p * DC + j * 16 + brow) * HP + k * 16 + bcol);
#pragma unroll
              for (int i = 0; i < 4; i++) f[p][4 * j + i] = w[i];
            }
        };
        load(Ks);
        mma_parts(r, rs, a, f);
        load(Qs);
        mma_parts(y, ys, a, f);
      }
    }
    if (lane == 0) dn::mbar_arrive(q_free);
    if (warp == 0 && c + 1 < chunks) {      // K of the next chunk over that of the one before
      if (c > 0) dn::mbar_wait(k_free, (c - 1) & 1, err);
      __syncwarp();
      part(sK + ((c + 1) & 1) * KB, c + 1, 0, &k_full[(c + 1) & 1]);
    }
    // What the halves exchange has one place a warp, and the partner has read the chunk before's: T comes behind t_free, on which every warp arrives after that.
    // (The wait costs nothing, the copy is under way since the chunk before; a second place would leave room for one block of 32 columns an SM.)
    dn::mbar_wait(t_full, c & 1, err);
    __syncwarp();
    // (the sums of the small parts' products join at the end: the fewer additions of full size, the fewer roundings)
    float out[2][4], osm[2][4];      // the outputs of tokens 16 hf ..
    {
      float* mine = xch + warp * DC_XCH * 32 + lane;
      const float* other = xch + (cg + (hf ^ 1) * CG) * DC_XCH * 32 + lane;
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) mine[(4 * i + j) * 32] = r[i][j] + rs[i][j];
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
          mine[(16 + 4 * i + j) * 32] = hf ? y[i][j] + ys[i][j] : y[2 + i][j] + ys[2 + i][j];
          out[i][j] = hf ? y[2 + i][j] : y[i][j];
          osm[i][j] = hf ? ys[2 + i][j] : ys[i][j];
        }
      asm volatile("bar.sync %0, 64;" ::"r"(1 + cg) : "memory");
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) r[i][j] = (r[i][j] + rs[i][j]) + other[(4 * i + j) * 32];
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) out[i][j] += other[(16 + 4 * i + j) * 32];
    }
    // V - G K S0
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const float2 gt = *reinterpret_cast<const float2*>(gm + 8 * i + 2 * (lane & 3));
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int t = 8 * i + 2 * (lane & 3) + (j & 1);
        r[i][j] = t < cnt ? fmaf(-((j & 1) ? gt.y : gt.x), r[i][j], Vs[t * VP + col + (j < 2 ? 0 : 8)]) : 0.f;
      }
    }
    int bad = first_not_finite([&](int i) -> float (&)[4] { return r[i]; }, lane, DC_ALL_FINITE);
    // U = T (..): tokens from 16 on alone see those from 16 on
    auto tile16 = [&](const bf16* m, int j, int k, uint32_t (&f)[3][4]) {      // tokens 16 j .. of T or A, places 16 k ..
#pragma unroll
      for (int p = 0; p < 3; p++) ldsm_x4(f[p], m + (p * DC + j * 16 + brow) * DC_TP + k * 16 + bcol);
    };
    float u[2][2][4];
    {
      float small[2][2][4];
      uint32_t a[3][4], f[3][4];
#pragma unroll
      for (int j = 0; j < 2; j++) { zero_tiles(u[j]); zero_tiles(small[j]); }
      a_frag(r[0], r[1], a);
      tile16(Ts, 0, 0, f);
      mma_parts(u[0], small[0], a, f);
      tile16(Ts, 1, 0, f);
      mma_parts(u[1], small[1], a, f);
      a_frag(r[2], r[3], a);
      tile16(Ts, 1, 1, f);
      mma_parts(u[1], small[1], a, f);
#pragma unroll
      for (int j = 0; j < 2; j++)
#pragma unroll
        for (int i = 0; i < 2; i++) {
          const float2 bt = *reinterpret_cast<const float2*>(gm + 2 * DC + 16 * j + 8 * i + 2 * (lane & 3));
#pragma unroll
          for (int x = 0; x < 4; x++) u[j][i][x] = fmaf((x & 1) ? bt.y : bt.x, r[2 * j + i][x], u[j][i][x] + small[j][i][x]);
        }
    }
    bad = first_not_finite([&](int i) -> float (&)[4] { return u[i >> 1][i & 1]; }, lane, bad);      // (T's rows, where a key, a decay or beta is the cause)
    if (warp == 1 && c + 1 < chunks) {
      dn::mbar_wait(q_free, c & 1, err);
      __syncwarp();
      part(sQ, c + 1, 1, q_full);
    }
    // O = .. + A U
    {
      const bf16* As = Ts + 3 * DC * DC_TP;
      float d[2][4], small[2][4];
      uint32_t a[3][4], f[3][4];
      zero_tiles(d);
      zero_tiles(small);
      a_frag(u[0][0], u[0][1], a);
      tile16(As, hf, 0, f);
      mma_parts(d, small, a, f);
      if (hf) {
        a_frag(u[1][0], u[1][1], a);
        tile16(As, 1, 1, f);
        mma_parts(d, small, a, f);
      }
      float* od = o + (size_t)n0 * Cv + (size_t)h * dv + col0 + col;
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const float2 gt = *reinterpret_cast<const float2*>(gm + 16 * hf + 8 * i + 2 * (lane & 3));
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const int t = 16 * hf + 8 * i + 2 * (lane & 3) + (j & 1);
          const float gj = (j & 1) ? gt.y : gt.x;
          if (t < cnt && (j < 2 ? okA : okB))
            od[(size_t)t * Cv + (j < 2 ? 0 : 8)] = t < (j < 2 ? bad & 255 : bad >> 8) ? fmaf(out[i][j], gj, d[i][j]) + fmaf(osm[i][j], gj, small[i][j]) : __int_as_float(0x7fffffff);
        }
      }
    }
    // S = G_32 S0 + (D_32 U)^T K.  The parts hold D_32 U as it is, not rounded to fp32
    uint32_t a[2][3][4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const float2 d = *reinterpret_cast<const float2*>(gm + DC + 8 * i + 2 * (lane & 3));
      const float (&x)[4] = u[i >> 1][i & 1];
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const float px = x[2 * j] * d.x, py = x[2 * j + 1] * d.y;
        uint32_t p[3];
        split3(px, py, p, fmaf(x[2 * j], d.x, -px), fmaf(x[2 * j + 1], d.y, -py));
#pragma unroll
        for (int z = 0; z < 3; z++) a[i >> 1][z][2 * (i & 1) + j] = p[z];
      }
    }
    const float gl = gm[DC - 1];
    __syncwarp();
    if (lane == 0) dn::mbar_arrive(t_free);
#pragma unroll
    for (int i = 0; i < DK / 64; i++) {      // 32 state rows: all products in one chain, the small ones first
      float d[4][4];
      uint32_t f[2][3][8];
      zero_tiles(d);
#pragma unroll
      for (int k = 0; k < 2; k++) {
#pragma unroll
        for (int p = 0; p < 3; p++)
#pragma unroll
          for (int j = 0; j < 2; j++) {
            uint32_t w[4];
            ldsm_x4_t(w, Ks + (p * DC + k * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)) * HP + i * 32 + j * 16 + (lane >> 4) * 8);
#pragma unroll
            for (int q = 0; q < 4; q++) f[k][p][4 * j + q] = w[q];
          }
        mma_small(d, a[k], f[k]);
      }
#pragma unroll
      for (int k = 0; k < 2; k++)
#pragma unroll
        for (int n = 0; n < 4; n++) dc_mma(d[n], a[k][0], f[k][0][2 * n], f[k][0][2 * n + 1]);
#pragma unroll
      for (int n = 0; n < 4; n++)
#pragma unroll
        for (int j = 0; j < 4; j++) S[4 * i + n][j] = fmaf(S[4 * i + n][j], gl, d[n][j]);
    }
    if (bad != DC_ALL_FINITE)
#pragma unroll
      for (int i = 0; i < NT; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
          if ((j < 2 ? bad & 255 : bad >> 8) < DC) S[i][j] = __int_as_float(0x7fffffff);
    __syncwarp();
    if (lane == 0) dn::mbar_arrive(k_free);
    if (warp == 2 && c + 1 < chunks) {
      dn::mbar_wait(t_free, c & 1, err);
      __syncwarp();
      rest(c + 1);
    }
  }
#pragma unroll
  for (int i = 0; i < NT; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int d = 8 * i + 2 * (lane & 3) + (j & 1);
      if (j < 2 ? okA : okB) Sg[(size_t)d * dv + (j < 2 ? 0 : 8)] = S[i][j];
    }
}

}  // namespace dnseq
