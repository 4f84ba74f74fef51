// Gated feed-forward rows of the hybrid decoders: out[t, c] = silu(x w_gate[c]) * (x w_up[c]), bf16 operands and result, fp32 sums.
//
// The dense GEMM of CTA pairs (dense_gemm_tc.cuh) with the activation in its epilogue.  As a library product with fp32 results and a pass
// over them this is 2 x 4 bytes per element of [T, 2 ff] more through memory: 3001 rows of 2048 -> 5632, 114 + 26 us there.
#include "dense_gemm_tc.cuh"

namespace b200 {

// w [2 ff, K]: gate rows, then up rows.  false: not taken (few rows, other types, sizes or alignments).
bool launch_dense_gated(const void* x, const void* w, void* out, int T, int ff, int K, int dt, cudaStream_t st) {
  if (dt != 0 || T <= dg::kBM || K % dg::kBK != 0 || ff % 8 != 0) return false;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(out)) & 15) return false;
  return dg::launch_cfg<256, 2, false, false, false, true>(x, w, out, nullptr, T, 2 * ff, K, st);
}

}  // namespace b200
