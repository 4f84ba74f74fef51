// What moe.cu and moe_tc.cu share.
#pragma once
#include <algorithm>

#include "seqmix.cuh"

namespace b200 {

// act of a gated expert from its gate and up products; ACT 3: clamped
template <int ACT>
__device__ __forceinline__ float expert_gate(float g, float u, const b200_expert_act& p) {
  if (ACT != 3) return seqmix::silu_exact(g) * u;
  g = fminf(g, p.limit);
  u = fminf(fmaxf(u, -p.limit), p.limit);
  return g / (1.f + expf(-p.alpha * g)) * (u + p.up_add);
}

// A grouped product in bf16 on the tensor cores (act_kind as ACT in moe.cu).  Token rows (act_kind != 0) are first copied to
// `rows` [pairs, K] in bucket order.  false: sizes or alignment it does not take, or no space for the rows.
bool grouped_linear_tc(int act_kind, void* out, const void* a, const void* w, const int32_t* off, const int32_t* pair_of_slot,
                       void* rows, int pairs, int top, int E, int K, int N, const b200_expert_act& act, cudaStream_t st);

}  // namespace b200
