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
// The merge of split keys, one block per token and head, right after launch_attn_tc.  Few blocks start under the attention's end (as dependents of
// it); more would all wait on the SMs that the attention leaves idle, and then share those.  us, plain and as dependents: one token over
// 2047 latent keys, 32 blocks, 24.9 and 22.8, four tokens, 128 blocks, 26.6 and 30.2; 8 tokens over 2048 keys, 256 blocks, 24.7 and 26.1.
template <typename... P, typename... A>
inline void launch_attn_merge(void (*kern)(P...), int blocks, int threads, cudaStream_t st, A... args) {
  if (blocks <= 64) launch_pdl(kern, dim3(blocks), dim3(threads), 0, st, args...);
  else kern<<<blocks, threads, 0, st>>>(static_cast<P>(args)...);
  B200_CUDA_LAUNCH_CHECK();
}

}  // namespace b200
