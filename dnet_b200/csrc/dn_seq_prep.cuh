// dn_seq_prep.cuh -- what lies between a mixer's projections and its scores or its recurrence, for runs of tokens (bf16), libdnet_b200_seq.so:
// short convolution, norm, rotation, cache append (attention); short convolution, SiLU, norm, gates (delta rule).
//
// Bound by latency: 2,048 tokens of 4,096 + 2 x 1,024 channels are 25 MB in and 25 out (50 for the delta rule, whose outputs are fp32) and take 32 and 43 us, 1.6 and
// 1.7 TB/s, a quarter of the memory's rate: what a block loads, and then what its norm needs, are two ways from memory one behind the other.  A block takes TOK neighbouring
// tokens and a thread 16 bytes of adjacent channels of all of them, so that a channel's convolution weights and input rows are read, and unpacked, once for TOK tokens, and holds
// its numbers in registers from the convolution to the store: a thread's channels lie in one head, and so do the pairs that rotate together.  Two tokens leave room for
// two blocks of 512 threads an SM; four, which read less, hold twice the registers and run alone: 39.5 and 54 us.  (Rows unpacked for every tap and token, the norm's
// root by every thread, cosines one by one: 72 instructions a channel and 58 and 69 us with four tokens; a block a token that read four rows and all weights for each and passed
// its numbers through shared memory: 87 and 96.)
// FEW: steps of no more tokens than SMs, a block of one token an SM: all registers and one path through the convolution, since such a block waits for its code and its loads (single
// tokens of 3,072 channels, four taps, in a decode step: attention 7.9 us without, 6.6 so; delta rule 7.3 and 6.6).
// Every token's numbers are formed in the same order whatever TOK is and whichever tokens come with it.
#pragma once
#include "dn_seq_kernels.cuh"

namespace dnseq {

constexpr int RUN_VECS = 2, RUN_MAX_TAPS = CONV_MAX_TAPS, RUN_MAX_ROT = 128;      // 16-byte channel groups of a thread; rotated dims of a head
constexpr int RUN_TOK = 2;                                                         // tokens of a block where run_tok says so, else one
// Two tokens a block read less and run longer, so that they pay once the blocks of single tokens queue.  us of one / two tokens a block, four taps:
//   attention, 1,536 channels: 400 tokens 6.8 / 7.5, 800 7.4 / 7.5, 1,000 10.7 / 8.0; 3,072 channels: 400 7.7 / 8.3, 600 11.5 / 10.4, 2,048 24.7 / 20.9;
//     6,144 channels: 200 9.8 / 11.4, 300 13.6 / 12.5, 2,048 44.3 / 32.4                  -> more than 1,024 threads an SM
//   delta rule, 1,536 and 3,072 channels (one pass of a block): 800 tokens 8.9 / 9.3 and 14.0 / 15.0, 1,000 12.0 / 9.7 and 18.2 / 15.7; 6,144 channels (two):
//     200 11.0 / 12.1, 300 16.7 / 15.0, 2,048 54.8 / 42.0                                 -> more than 2,300 threads an SM, 1,024 with more than 4,096 channels
constexpr int RUN_ATTN_FROM = 1024, RUN_DELTA_FROM = 2300, RUN_DELTA_WIDE_FROM = 1024, RUN_DELTA_CHANNELS = 4096;
inline int run_tok(int tokens, int threads, int sms, int from) { return (long long)tokens * threads > (long long)sms * from ? RUN_TOK : 1; }

// whether no convolution of the block's tokens reaches behind the first row of an entry (nor the last token of the step)
template <int TAPS, int TOK>
__device__ __forceinline__ bool run_plain(const int (&local)[TOK], int n0, int N, bool carry) {
  return !carry && local[0] >= TAPS - 1 && local[TOK - 1] - local[0] == TOK - 1 && n0 + TOK <= N;
}
// x = the convolution of channels c .. c + 7 (offset `off` among the carried ones) for the block's tokens; U [N][ldu]
template <int TAPS, int TOK>
__device__ __forceinline__ void conv_run(const bf16* __restrict__ U, int ldu, const bf16* __restrict__ cw, int c, int n0, int N, const int (&local)[TOK], bf16* const (&st)[TOK], int off,
                                         int ldst, bool carry, bool plain, float (&x)[TOK][8]) {
  constexpr int B = TAPS > 0 ? TAPS - 1 : 0;      // rows in front of a token
  uint4 row[TOK + B];
#pragma unroll
  for (int r = 0; r < TOK + B; r++) {
    const int n = n0 - B + r;
    row[r] = make_uint4(0u, 0u, 0u, 0u);
    if (n < N && B - r <= local[0]) row[r] = *reinterpret_cast<const uint4*>(U + (size_t)n * ldu + c);      // (rows of other entries are left out below)
  }
  if constexpr (TAPS == 0) {
#pragma unroll
    for (int i = 0; i < TOK; i++) ldv(reinterpret_cast<const bf16*>(&row[i]), x[i]);
  } else if (plain) {      // every row is one of the step's: a row's numbers are unpacked once for all the tokens that it meets
    uint4 wv[TAPS];      // [8 channels][TAPS]
#pragma unroll
    for (int j = 0; j < TAPS; j++) wv[j] = *reinterpret_cast<const uint4*>(cw + (size_t)c * TAPS + j * 8);
    const bf16* wb = reinterpret_cast<const bf16*>(wv);
#pragma unroll
    for (int h = 0; h < 4; h++) {      // two channels
      float2 w[TAPS], v[TOK + B];
#pragma unroll
      for (int j = 0; j < TAPS; j++) w[j] = make_float2(__bfloat162float(wb[2 * h * TAPS + j]), __bfloat162float(wb[(2 * h + 1) * TAPS + j]));
#pragma unroll
      for (int r = 0; r < TOK + B; r++) v[r] = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(&row[r])[h]);
#pragma unroll
      for (int i = 0; i < TOK; i++) {
        float2 a = make_float2(0.f, 0.f);
#pragma unroll
        for (int j = 0; j < TAPS; j++) a = fma2(w[j], v[i + j], a);
        x[i][2 * h] = a.x;
        x[i][2 * h + 1] = a.y;
      }
    }
  } else {
    float wl[8 * TAPS];
    canon_weights<bf16, TAPS>(cw, c, wl);
#pragma unroll
    for (int i = 0; i < TOK; i++) {
      uint4 in[TAPS];
#pragma unroll
      for (int j = 0; j < TAPS; j++) {
        const int back = TAPS - 1 - j;
        in[j] = row[i + j];
        if (back > local[i] && n0 + i < N) in[j] = *reinterpret_cast<const uint4*>(st[i] + (size_t)(TAPS - 1 - (back - local[i])) * ldst + off + c);
      }
#pragma unroll
      for (int e = 0; e < 8; e++) x[i][e] = 0.f;
#pragma unroll
      for (int j = 0; j < TAPS; j++) {
        float v[8];
        ldv(reinterpret_cast<const bf16*>(&in[j]), v);
#pragma unroll
        for (int e = 0; e < 8; e++) x[i][e] += wl[e * TAPS + j] * v[e];
      }
      if (carry && n0 + i < N)      // the only token of its entry: its input takes its place among the carried ones (places beyond N hold the last token's slot)
#pragma unroll
        for (int j = 1; j < TAPS; j++) *reinterpret_cast<uint4*>(st[i] + (size_t)(j - 1) * ldst + off + c) = in[j];
    }
  }
}

// k_attn_prep for projections normed as a whole (or not at all) whose pairs (2 i, 2 i + 1) rotate.  Head sizes in whole 16 bytes.
template <int TAPS, int TOK, bool FEW = false>
__global__ void __launch_bounds__(512, FEW ? 1 : 2) k_attn_prep_run(AttnPrep a, Batch b, const bf16* __restrict__ Uq, const bf16* __restrict__ Uk, const bf16* __restrict__ Uv,
                                                       const bf16* __restrict__ cwq, const bf16* __restrict__ cwk, const bf16* __restrict__ cwv, const bf16* __restrict__ nq,
                                                       const bf16* __restrict__ nk, bf16* __restrict__ cstate, size_t slot_stride, bf16* __restrict__ qout,
                                                       bf16* __restrict__ kpool, bf16* __restrict__ vpool) {
  __shared__ __align__(16) float cst[TOK][RUN_MAX_ROT / 2], snt[TOK][RUN_MAX_ROT / 2];
  __shared__ float red[2 * TOK][16], tot[2 * TOK];
  const int Cq = a.H * a.dk, Ck = a.own_kv ? a.G * a.dk : 0, Cv = (a.own_kv && a.own_v) ? a.gv * a.dv : 0, ldst = Cq + Ck + Cv;
  const int n0 = blockIdx.x * TOK, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int local[TOK], pos[TOK];
  size_t cache[TOK];      // row of the cache
  bf16* st[TOK];
#pragma unroll
  for (int i = 0; i < TOK; i++) {
    const int n = min(n0 + i, b.N - 1), slot = b.slot[n];
    pos[i] = b.pos[n];
    local[i] = n - b.first[n];
    cache[i] = (size_t)b.bt[(size_t)slot * b.max_pages + pos[i] / PAGE] * PAGE + pos[i] % PAGE;
    st[i] = cstate + (size_t)slot * slot_stride;
  }
  const bool plain = !FEW && run_plain<TAPS, TOK>(local, n0, b.N, a.carry != 0);
  float x[RUN_VECS][TOK][8], sq[TOK], sk[TOK];
#pragma unroll
  for (int i = 0; i < TOK; i++) sq[i] = sk[i] = 0.f;
#pragma unroll
  for (int u = 0; u < RUN_VECS; u++) {
    const int c = (threadIdx.x + u * blockDim.x) * 8;
    if (c >= ldst) continue;
    const int z = c < Cq ? 0 : c < Cq + Ck ? 1 : 2, off = z == 0 ? 0 : z == 1 ? Cq : Cq + Ck;
    conv_run<TAPS, TOK>(z == 0 ? Uq : z == 1 ? Uk : Uv, z == 0 ? Cq : z == 1 ? Ck : Cv, z == 0 ? cwq : z == 1 ? cwk : cwv, c - off, n0, b.N, local, st, off, ldst, a.carry != 0, plain, x[u]);
#pragma unroll
    for (int i = 0; i < TOK; i++) {
      if (z == 2) {
        if (n0 + i < b.N) stv(vpool + cache[i] * Cv + (c - off), x[u][i]);
        continue;
      }
      float s = z ? sk[i] : sq[i];
#pragma unroll
      for (int e = 0; e < 8; e++) s += x[u][i][e] * x[u][i][e];
      if (z) sk[i] = s; else sq[i] = s;
    }
  }
  const int hr = a.rot / 2;
  for (int e = threadIdx.x; e < TOK * hr; e += blockDim.x) {
    const int i = e / hr, d = e - i * hr;
    float sn, cs;
    sincosf((float)b.pos[min(n0 + i, b.N - 1)] * a.inv_freq[d], &sn, &cs);
    cst[i][d] = cs * a.mscale;
    snt[i][d] = sn * a.mscale;
  }
  if (a.norm) {      // sums over the block, warp by warp
#pragma unroll
    for (int k = 0; k < 2 * TOK; k++) {
      const float v = warp_sum(k < TOK ? sq[k % TOK] : sk[k % TOK]);
      if (lane == 0) red[k][warp] = v;
    }
  }
  __syncthreads();
  if (a.norm) {
    for (int k = warp; k < 2 * TOK; k += nw) {
      const float t = warp_sum(lane < nw ? red[k][lane] : 0.f);
      if (lane == 0) tot[k] = 1.f / sqrtf(t / (float)(k < TOK ? Cq : Ck) + a.eps);      // (once a token, not by every thread)
    }
    __syncthreads();
  }
  const bool nvec = (((uintptr_t)nq | (uintptr_t)nk) & 15) == 0;      // (norm weights may lie at any address)
#pragma unroll
  for (int u = 0; u < RUN_VECS; u++) {
    const int c = (threadIdx.x + u * blockDim.x) * 8;
    if (c >= Cq + Ck) continue;
    const bool isq = c < Cq;
    const int cc = isq ? c : c - Cq, d = cc % a.dk;
    float w[8];
    if (a.norm) {
      const bf16* wp = (isq ? nq : nk) + cc;
      if (nvec) ldv(wp, w);
      else
#pragma unroll
        for (int e = 0; e < 8; e++) w[e] = ldf(wp + e);
    }
#pragma unroll
    for (int i = 0; i < TOK; i++) {
      if (n0 + i >= b.N) continue;
      float (&y)[8] = x[u][i];
      if (a.norm) {
        const float r = tot[isq ? i : TOK + i];
#pragma unroll
        for (int e = 0; e < 8; e++) y[e] = y[e] * r * w[e];
      }
      if (d < a.rot) {      // (the angles' room ends on a boundary of four; pairs from rot on are left)
        const float4 c4 = *reinterpret_cast<const float4*>(&cst[i][d / 2]), s4 = *reinterpret_cast<const float4*>(&snt[i][d / 2]);
        const float cc[4] = {c4.x, c4.y, c4.z, c4.w}, ss[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
        for (int e = 0; e < 8; e += 2)
          if (d + e + 1 < a.rot) {
            const float cs = cc[e / 2], sn = ss[e / 2], y0 = y[e] * cs - y[e + 1] * sn, y1 = y[e + 1] * cs + y[e] * sn;
            y[e] = y0; y[e + 1] = y1;
          }
      }
      if (isq) {
        if (a.qt_every > 0) {
          const float qt = 1.f + a.qt_coef * logf((float)((pos[i] + 1) / a.qt_every + 1));
#pragma unroll
          for (int e = 0; e < 8; e++) y[e] *= qt;
        }
        stv(qout + (size_t)(n0 + i) * Cq + cc, y);
      } else stv(kpool + cache[i] * Ck + cc, y);
    }
  }
}

// k_delta_prep for key sizes of 8, 16, .. 256: a head's sum of squares runs over a thread's eight channels, then pairwise over the head's lanes
template <int TAPS, int TOK, bool FEW = false>
__global__ void __launch_bounds__(512, FEW ? 1 : 2) k_delta_prep_run(DeltaPrep a, Batch b, const bf16* __restrict__ Uq, const bf16* __restrict__ Uk, const bf16* __restrict__ Uv,
                                                        const bf16* __restrict__ cwq, const bf16* __restrict__ cwk, const bf16* __restrict__ cwv, const float* __restrict__ pa,
                                                        const float* __restrict__ pb, const bf16* __restrict__ A_log, const bf16* __restrict__ dt_bias,
                                                        bf16* __restrict__ cstate, size_t slot_stride, float* __restrict__ qn, float* __restrict__ kn,
                                                        float* __restrict__ vv, float* __restrict__ beta, float* __restrict__ decay) {
  const int Cq = a.G * a.dk, Cv = a.H * a.dv, ldst = 2 * Cq + Cv, n0 = blockIdx.x * TOK, lanes = a.dk / 8;
  int local[TOK];
  bf16* st[TOK];
#pragma unroll
  for (int i = 0; i < TOK; i++) {
    const int n = min(n0 + i, b.N - 1);
    local[i] = n - b.first[n];
    st[i] = cstate + (size_t)b.slot[n] * slot_stride;
  }
  const bool plain = !FEW && run_plain<TAPS, TOK>(local, n0, b.N, false);
  for (int base = 0; base < ldst; base += blockDim.x * 8) {
    const int c = base + threadIdx.x * 8, z = c < Cq ? 0 : c < 2 * Cq ? 1 : 2, off = z * Cq;
    const bool in = c < ldst;
    float x[TOK][8];
    if (in) conv_run<TAPS, TOK>(z == 0 ? Uq : z == 1 ? Uk : Uv, z == 2 ? Cv : Cq, z == 0 ? cwq : z == 1 ? cwk : cwv, c - off, n0, b.N, local, st, off, ldst, false, plain, x);
#pragma unroll
    for (int i = 0; i < TOK; i++) {
      float ss = 0.f;
#pragma unroll
      for (int e = 0; e < 8; e++) {
        x[i][e] = in ? silu_f(x[i][e]) : 0.f;
        ss += x[i][e] * x[i][e];
      }
      for (int o = lanes / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if (!in || n0 + i >= b.N) continue;
      float* dst = z == 2 ? vv + (size_t)(n0 + i) * Cv + (c - off) : (z ? kn : qn) + (size_t)(n0 + i) * Cq + (c - off);
      const float r = z == 2 ? 1.f : (1.f / sqrtf(ss + 1e-6f)) * (z == 0 ? 1.f / sqrtf((float)a.dk) : 1.f);
#pragma unroll
      for (int e = 0; e < 8; e += 4) *reinterpret_cast<float4*>(dst + e) = make_float4(x[i][e] * r, x[i][e + 1] * r, x[i][e + 2] * r, x[i][e + 3] * r);
    }
  }
  for (int e = threadIdx.x; e < TOK * a.H; e += blockDim.x) {
    const int n = n0 + e / a.H, h = e % a.H;
    if (n >= b.N) break;
    beta[(size_t)n * a.H + h] = 1.f / (1.f + expf(-pb[(size_t)n * a.H + h]));
    decay[(size_t)n * a.H + h] = expf(-expf(ldf(A_log + h)) * softplus_f(pa[(size_t)n * a.H + h] + ldf(dt_bias + h)));
  }
}

}  // namespace dnseq
