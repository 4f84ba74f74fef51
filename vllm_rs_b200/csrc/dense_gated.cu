// Gated feed-forward rows of the hybrid decoders: out[t, c] = silu(x w_gate[c]) * (x w_up[c]), bf16 operands and result, fp32 sums.
//
// The dense GEMM of CTA pairs (dense_gemm_tc.cuh) with the activation in its epilogue.  As a library product with fp32 results and a pass
// over them this is 2 x 4 bytes per element of [T, 2 ff] more through memory: 3001 rows of 2048 -> 5632, 114 + 26 us there.
#include <cmath>

#include "dense_gemm_tc.cuh"

namespace b200 {

// Whether launch_dense_gated is faster than the library and a pass over its results, on `pairs` pairs of SMs.  A pair takes its tiles of
// 256 rows and 128 channels in turn; the library cuts finer, so what decides is how much of the last turn is work.  Turns it takes
// the library for the same work against turns here, plus either one's start: lines through 264 measured sizes, T 129 - 3001, ff 256 - 11008, K 1024 -
// 4096, of which this rule takes 1.03 times the faster one once (this kernel alone 1.6 times on average, 3 at most; the library
// alone 1.024).  us, here and there: 2048 -> 512, 300 rows 19.3 / 7.6; -> 5632, 256 rows 23.4 / 17.1, 1000 rows 41.3 / 46.2, 3001 rows 101 / 141;
// 1024 -> 5632, 1000 rows 34.5 / 31.9, 3001 rows 81 / 94.
bool dense_gated_pays(int T, int ff, int K, int pairs) {
  const double tile_rows = 2 * dg::kBM, tile_cols = 128;
  const double turns = std::ceil(std::ceil(T / tile_rows) * std::ceil(ff / tile_cols) / pairs);
  const double work = T / tile_rows * (ff / tile_cols) / pairs;
  return turns >= 2 && work > (K < 2048 ? 0.28 + 0.78 * turns : 0.14 + 0.72 * turns);
}

// w [2 ff, K]: gate rows, then up rows.  false: not taken (few rows, other types, sizes or alignments).
bool launch_dense_gated(const void* x, const void* w, void* out, int T, int ff, int K, int dt, cudaStream_t st) {
  if (dt != 0 || T <= dg::kBM || K % dg::kBK != 0 || ff % 8 != 0) return false;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(out)) & 15) return false;
  return dg::launch_cfg<256, 2, false, false, false, true>(x, w, out, nullptr, T, 2 * ff, K, st);
}

}  // namespace b200
