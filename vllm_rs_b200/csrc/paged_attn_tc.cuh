// Softmax attention of the hybrid decoders on tcgen05 tensor cores (paged_attn_tc.cu): what window_attn.cu and latent_attn.cu
// hand to it.
#pragma once
#include "seqmix.cuh"

namespace b200 {

// A step's attention over paged caches of bf16 rows.  Query head h belongs to key head h / group and reads value head
// (h / group) % v_heads.  The values are a cache of their own, or (v_cache == NULL) the first vdim entries of the key rows.
struct AttnTcProblem {
  void* out;                       // [T, heads, vdim] bf16, or fp32 with out_f32
  const float* q;                  // [T, heads, dim]
  const void* k_cache;             // [pages, 64, kv_heads, dim]
  const void* v_cache;             // [pages, 64, v_heads, vdim] or NULL
  const float* sink;               // [heads] or NULL
  const float* gate;               // logits [T, ld_gate]: one per head, or per element with gate_elems; or NULL
  int ld_gate, gate_elems;
  const uint32_t *cu, *ctx, *block_tables;
  int max_blocks, num_seqs, T, heads, kv_heads, v_heads, dim, vdim;
  int window, keep_first, chunk;
  float scale, softcap;
  const float* slopes;             // [heads] or NULL
  const float* dist_bias;          // [heads, dist_n] or NULL
  int dist_n, out_f32;
  int nsplit;                      // key splits; > 1: unnormalised parts [T, heads, nsplit, vdim] and (max, sum) pairs
  float *part_o, *part_ml;
};
// steps of few rows (decoding): the keys of a row are split over several blocks
inline bool attn_few_rows(int T) { return T <= 2 * sm_count() / 4; }
// whether these sizes and pointers are taken (bf16 caches only)
bool attn_tc_takes(const AttnTcProblem& p);
// key splits that fill the chip for a step of T rows of which every sequence brings few (1: no split); max_blocks: pages of the
// longest context, 0 where that is not known
int attn_tc_splits(int T, int kv_heads, int vdim, int shared_kv, int window, int keep_first, int max_blocks);
void launch_attn_tc(const AttnTcProblem& p, cudaStream_t st);

}  // namespace b200
