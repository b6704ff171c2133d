// dn_seq_attn_prompt.cuh -- plain softmax attention of the layer-list models' prompt portions (libdnet_b200_seq.so, bf16, head size 128) on k_attn_prompt
// (dn_attn_prompt.cuh): what a row block of a ragged batch is, and which layers and steps take it.
#pragma once
#include "dn_attn_prompt.cuh"
#include "dn_seq_kernels.cuh"

namespace dnseq {

constexpr int AB_MAX_ENTRIES = 64;      // (a block is found by walking the entries)

// The row blocks of a step's entries, one entry after the other; pages [page][64][key heads x 128] of keys and of values
struct ApBatch {
  Batch b;
  int chunk, window;      // the mask (attn_lo)
  static constexpr bool RISING = false;
  __device__ __forceinline__ void start() {}
  __device__ __forceinline__ int blocks(int TB) const {
    int n = 0;
    for (int e = 0; e < b.E; e++) n += (b.ent_start[e + 1] - b.ent_start[e] + TB - 1) / TB;
    return n;
  }
  __device__ __forceinline__ dn::ApBlock block(int i, int TB) const {
    int e = 0, s = b.ent_start[0], n = b.ent_start[1] - s;
    while (i >= (n + TB - 1) / TB && e + 1 < b.E) {
      i -= (n + TB - 1) / TB;
      s += n;
      e++;
      n = b.ent_start[e + 1] - s;
    }
    dn::ApBlock r;
    r.row0 = s + i * TB;
    r.nq = min(TB, n - i * TB);
    r.p_first = b.ent_pos0[e] + i * TB;
    r.page0 = attn_lo(r.p_first, chunk, window) / PAGE;
    r.pages = (r.p_first + r.nq + PAGE - 1) / PAGE;
    r.bt = b.bt + (size_t)b.ent_slot[e] * b.max_pages;
    return r;
  }
  __device__ __forceinline__ int lo(int pos) const { return attn_lo(pos, chunk, window); }
  __device__ __forceinline__ void at(int page, int kvh, int, int half, int& c0, int& c1) const { c0 = kvh * 128 + half * 64; c1 = page * PAGE; }
};

}  // namespace dnseq
