// dn_attn_few.cuh -- causal attention of a few query tokens (up to FEW_ROWS rows of a key head's group) over the paged 16-bit KV cache,
// libdnet_b200.so: single tokens outside the step kernel, drafts, the end of a chunked prompt.
//
// Bound by latency behind short contexts and by reading the keys and values behind long ones.  A CTA takes one key / value head, all rows of its
// group (row = token x G + head) and a run of key tiles (128 keys, two pages); the tiles are dealt out over as many CTAs as fill the SMs, FEW_SPLITS a key
// head at most (one or two key heads leave SMs idle), whose partial outputs the last one to finish (an atomic count, nobody waits) joins in the order of the keys.  A tile comes by asynchronous copies, the next
// one while it is worked on; each of the eight warps takes 16 of its keys for each 16 rows, on mma.sync:
//   S = Q K^T   Q stays in registers
//   P V         a weight goes in three bf16 parts (all 24 bits of its mantissa), the scores' registers being the operand's as they lie
// Every MMA starts from zero or from the smaller parts, and sums meet in fp32 additions (an accumulator handed on is cut, not rounded, at each step).
// On the 128-row tiles of k_attn_prefill_tc one CTA a key head walked the tiles: 3 tokens behind 256, eight groups of 4, a layer 105.9 us, 96.0 so; one
// Mixtral-8x7B token behind 512 169.9 / 154.4; one token behind 8,192, eight groups of 4, a layer 133.7 / 106.4.  (One CTA an SM: 255 registers a thread hold the queries,
// the outputs and a tile's scores.)
#pragma once
#include "dn_attn_tc.cuh"

namespace dn {

constexpr int FEW_ROWS = 32, FEW_WARPS = 8, FEW_THREADS = FEW_WARPS * 32, FEW_KEYS = 128;
constexpr int FEW_SPLITS = 32;                                // CTAs that share a key head's tiles, at most
constexpr int FEW_PITCH = HD * 2 + 16;                        // bytes of a staged row: ldmatrix meets no bank twice
constexpr int FEW_STAGE = 2 * FEW_KEYS * FEW_PITCH;           // a tile's keys and values
constexpr int FEW_SMEM = 2 * FEW_STAGE + FEW_ROWS * FEW_PITCH;
constexpr int FEW_PART = 16 * (HD + 2);                       // floats of 16 rows' partial output: sums, references, outputs
static_assert(FEW_WARPS * FEW_PART * 4 <= 2 * FEW_STAGE, "the warps' outputs meet in the tiles' memory");

struct FewParams {
  const bf16 *q, *pool;          // [T][n_heads][128] (RoPE applied, unscaled); this layer's pages
  bf16* out;                     // [T][n_heads][128]
  const int32_t* block_table;
  const StepState* st;
  float* part;                   // [n_kv][splits][FEW_ROWS / 16][FEW_PART]
  unsigned int* count;           // [n_kv], zero between launches
  int n_heads, n_kv, G, T;
};

__device__ __forceinline__ void few_cp16(uint32_t dst, const void* src, bool have) {      // zeros where there is nothing
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(have ? 16 : 0) : "memory");
}
__device__ __forceinline__ void few_ldm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void few_ldm4t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void few_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, const float (&c)[4]) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}

// MT: tiles of 16 rows
template <int MT>
__global__ void __launch_bounds__(FEW_THREADS, 1) k_attn_few(const FewParams p) {
  extern __shared__ __align__(16) unsigned char few_smem[];
  __shared__ bool last_s;
  pdl_launch_dependents();
  pdl_wait();
  constexpr int WPM = FEW_WARPS / MT, KW = FEW_KEYS / WPM;      // warps of 16 rows; keys of a tile that a warp takes
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g8 = lane >> 2, t4 = lane & 3;
  const int kvh = blockIdx.x, z = blockIdx.y, rows = p.G * p.T;
  const int pos0 = p.st->pos, kv_len = pos0 + p.T, tiles = (kv_len + FEW_KEYS - 1) / FEW_KEYS;
  const int nz = min((int)gridDim.y, tiles);
  if (z >= nz) return;
  const int j0 = (int)((long long)tiles * z / nz), j1 = (int)((long long)tiles * (z + 1) / nz);
  const uint32_t sm = smem_u32(few_smem), smq = sm + 2 * FEW_STAGE;

  auto stage = [&](int j) {      // keys and values of tile j; a row is 16 pieces of 16 bytes
    const uint32_t dst = sm + ((j - j0) & 1) * FEW_STAGE;
    const int c = threadIdx.x & 15;
#pragma unroll
    for (int pg = 0; pg < 2; ++pg) {
      const int key0 = j * FEW_KEYS + pg * PAGE;
      const int phys = p.block_table[key0 < kv_len ? key0 / PAGE : 0];
      const bf16* k = p.pool + (((size_t)phys * 2) * p.n_kv + kvh) * (PAGE * HD) + c * 8;
      const bf16* v = k + (size_t)p.n_kv * (PAGE * HD);
#pragma unroll
      for (int i = 0; i < PAGE / 16; ++i) {
        const int r = i * 16 + (threadIdx.x >> 4);
        const bool have = key0 + r < kv_len;
        const uint32_t at = dst + (pg * PAGE + r) * FEW_PITCH + c * 16;
        few_cp16(at, k + r * HD, have);
        few_cp16(at + FEW_KEYS * FEW_PITCH, v + r * HD, have);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int i = threadIdx.x; i < MT * 16 * 16; i += FEW_THREADS) {
    const int r = i >> 4, c = i & 15;
    few_cp16(smq + r * FEW_PITCH + c * 16, p.q + ((size_t)(r < rows ? r / p.G : 0) * p.n_heads + kvh * p.G + (r < rows ? r % p.G : 0)) * HD + c * 8, r < rows);
  }
  stage(j0);

  const int mt = warp / WPM, wk = warp % WPM;      // this warp's rows; its place among the keys
  const int ra = mt * 16 + g8, rb = ra + 8;        // rows of the fragments
  const int last_a = ra < rows ? pos0 + ra / p.G : -1, last_b = rb < rows ? pos0 + rb / p.G : -1;      // last visible key
  const float sc2 = 0.08838834764831845f * LOG2E;
  uint32_t qf[8][4];
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, o[16][4];
#pragma unroll
  for (int i = 0; i < 16; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;

  for (int j = j0; j < j1; ++j) {
    if (j + 1 < j1) {
      stage(j + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (j == j0)
#pragma unroll
      for (int k = 0; k < 8; ++k) few_ldm4(qf[k], smq + (mt * 16 + (lane & 15)) * FEW_PITCH + k * 32 + (lane >> 4) * 16);
    const uint32_t sk = sm + ((j - j0) & 1) * FEW_STAGE, sv = sk + FEW_KEYS * FEW_PITCH;
#pragma unroll 1
    for (int h = 0; h < KW / 16; ++h) {
      const int r0 = wk * KW + h * 16, key0 = j * FEW_KEYS + r0;
      if (key0 >= kv_len) continue;
      float s[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f;
      const float zero[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k = 0; k < 8; k += 2)
#pragma unroll
        for (int i = 0; i < 2; ++i) {      // 8 keys x 32 dims
          uint32_t b[4];
          few_ldm4(b, sk + (r0 + i * 8 + (lane & 7)) * FEW_PITCH + k * 32 + (lane >> 3) * 16);
          float d[4], e[4];
          few_mma(d, qf[k], b[0], b[1], zero);
          few_mma(e, qf[k + 1], b[2], b[3], zero);
#pragma unroll
          for (int x = 0; x < 4; ++x) s[i][x] += d[x] + e[x];
        }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int x = 0; x < 4; ++x)
          if (key0 + i * 8 + 2 * t4 + (x & 1) > (x < 2 ? last_a : last_b)) s[i][x] = -INFINITY;
      float f[2];
#pragma unroll
      for (int y = 0; y < 2; ++y) {
        float mx = fmaxf(fmaxf(s[0][2 * y], s[0][2 * y + 1]), fmaxf(s[1][2 * y], s[1][2 * y + 1]));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float n = fmaxf(m[y], mx * sc2);
        f[y] = m[y] == n ? 1.f : exp2f(m[y] - n);      // 0 for a row that has seen nothing yet
        m[y] = n;
        const float nref = n == -INFINITY ? 0.f : -n;
        float sum = 0.f;
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            float& w = s[i][2 * y + x];
            w = tc_ex2(fmaf(w, sc2, nref));
            sum += w;
          }
        l[y] = fmaf(l[y], f[y], sum);
      }
      uint32_t pa[3][4];      // three parts, cut: rows g8, g8 + 8 of keys 2 t4 .., then of keys 8 + 2 t4 ..
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int y = 0; y < 2; ++y) {
          float2 w = make_float2(s[i][2 * y], s[i][2 * y + 1]);
#pragma unroll
          for (int part = 0; part < 3; ++part) {
            pa[part][2 * i + y] = upper_halves(w.x, w.y);
            if (part < 2) w = below_upper_halves(w);
          }
        }
#pragma unroll
      for (int n = 0; n < 8; ++n) {      // 16 keys x 16 dims
        uint32_t b[4];
        few_ldm4t(b, sv + (r0 + (lane & 15)) * FEW_PITCH + n * 32 + (lane >> 4) * 16);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          float d[4], e[4];
          few_mma(d, pa[2], b[2 * i], b[2 * i + 1], zero);
          few_mma(d, pa[1], b[2 * i], b[2 * i + 1], d);
          few_mma(e, pa[0], b[2 * i], b[2 * i + 1], zero);
          float (&a)[4] = o[2 * n + i];
#pragma unroll
          for (int x = 0; x < 4; ++x) a[x] = fmaf(a[x], f[x >> 1], e[x] + d[x]);
        }
      }
    }
    __syncthreads();      // the tile's memory may be written again
  }
#pragma unroll
  for (int y = 0; y < 2; ++y) {
    l[y] += __shfl_xor_sync(0xffffffffu, l[y], 1);
    l[y] += __shfl_xor_sync(0xffffffffu, l[y], 2);
  }
  // the warps' outputs meet: [warp][16 sums, 16 references, 16 x 128 outputs]
  float* wp = reinterpret_cast<float*>(few_smem) + warp * FEW_PART;
  if (t4 == 0) { wp[g8] = l[0]; wp[g8 + 8] = l[1]; wp[16 + g8] = m[0]; wp[24 + g8] = m[1]; }
#pragma unroll
  for (int n = 0; n < 16; ++n) {
    *reinterpret_cast<float2*>(wp + 32 + g8 * HD + n * 8 + 2 * t4) = make_float2(o[n][0], o[n][1]);
    *reinterpret_cast<float2*>(wp + 32 + (g8 + 8) * HD + n * 8 + 2 * t4) = make_float2(o[n][2], o[n][3]);
  }
  __syncthreads();
  auto store = [&](int row, int d, const float4& y, float L) {
    const float inv = 1.0f / L;
    uint2 w;
    w.x = pack_bf16x2(y.x * inv, y.y * inv);
    w.y = pack_bf16x2(y.z * inv, y.w * inv);
    *reinterpret_cast<uint2*>(p.out + ((size_t)(row / p.G) * p.n_heads + kvh * p.G + row % p.G) * HD + d) = w;
  };
  float* mine = p.part + (size_t)(kvh * gridDim.y + z) * MT * FEW_PART;
  for (int i = threadIdx.x; i < MT * 16 * 32; i += FEW_THREADS) {
    const int row = i >> 5, d = (i & 31) * 4, tile = row >> 4, r = row & 15;
    if (row >= rows) continue;
    const float* src = reinterpret_cast<const float*>(few_smem) + tile * WPM * FEW_PART;
    float M = -INFINITY, L = 0.f;
    float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int w = 0; w < WPM; ++w) M = fmaxf(M, src[w * FEW_PART + 16 + r]);
#pragma unroll
    for (int w = 0; w < WPM; ++w) {
      const float mi = src[w * FEW_PART + 16 + r], fi = mi == -INFINITY ? 0.f : exp2f(mi - M);
      const float4 a = *reinterpret_cast<const float4*>(src + w * FEW_PART + 32 + r * HD + d);
      L = fmaf(fi, src[w * FEW_PART + r], L);
      y.x = fmaf(fi, a.x, y.x); y.y = fmaf(fi, a.y, y.y); y.z = fmaf(fi, a.z, y.z); y.w = fmaf(fi, a.w, y.w);
    }
    if (nz == 1) store(row, d, y, L);
    else {
      float* dst = mine + tile * FEW_PART;
      __stcg(reinterpret_cast<float4*>(dst + 32 + r * HD + d), y);
      if (d == 0) { __stcg(dst + r, L); __stcg(dst + 16 + r, M); }
    }
  }
  if (nz == 1) return;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last_s = atomicAdd(p.count + kvh, 1u) == (unsigned int)nz - 1u;
    if (last_s) p.count[kvh] = 0u;      // (for the next launch)
    __threadfence();
  }
  __syncthreads();
  if (!last_s) return;
  // the splits' outputs, joined relative to the largest reference
  const size_t stride = (size_t)MT * FEW_PART;
  for (int i = threadIdx.x; i < MT * 16 * 32; i += FEW_THREADS) {
    const int row = i >> 5, d = (i & 31) * 4, r = row & 15;
    if (row >= rows) continue;
    const float* src = p.part + ((size_t)kvh * gridDim.y * MT + (row >> 4)) * FEW_PART;
    float M = -INFINITY, L = 0.f;
    for (int k = 0; k < nz; ++k) M = fmaxf(M, __ldcg(src + k * stride + 16 + r));
    float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int k = 0; k < nz; ++k) {
      const float mi = __ldcg(src + k * stride + 16 + r), fi = mi == -INFINITY ? 0.f : exp2f(mi - M);
      const float4 a = __ldcg(reinterpret_cast<const float4*>(src + k * stride + 32 + r * HD + d));
      L = fmaf(fi, __ldcg(src + k * stride + r), L);
      y.x = fmaf(fi, a.x, y.x); y.y = fmaf(fi, a.y, y.y); y.z = fmaf(fi, a.z, y.z); y.w = fmaf(fi, a.w, y.w);
    }
    store(row, d, y, L);
  }
}

}  // namespace dn
