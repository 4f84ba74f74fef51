// Dense fp16 GEMM on tcgen05 (SS mode): C[m, n] = A[m, k] x W[n, k]^T, fp32 accumulation in TMEM,
// fp16 or fp32 output, optional bias.
//
// Replaces the cuBLAS call behind Linear::forward (src/models/layers/linear.rs:75-123)
// for fp16 checkpoints (Llama-3-8B fp16 chunked prefill), the lm_head
// (src/models/llama.rs:311-320) and -- together with wna16_dequant_kernel below --
// the W4A16 / W8A16 linears of large prefill steps, where dequantising a layer's weights ONCE into an
// fp16 scratch and running this kernel beats re-dequantising them for every 256-token tile
// (the Marlin call of src/utils/gptq.rs:118-146 at M = thousands of tokens).
//
// Both operands are K-major, so both arrive through TMA (SWIZZLE_128B, 64-element K blocks) and
// feed tcgen05.mma.kind::f16 through shared-memory descriptors.  "P" is the operand whose rows
// become TMEM lanes (128 per CTA), "Q" the one whose rows become accumulator columns (BN per MMA):
//   prefill (M > 128):  P = activations, Q = weights, BN = 256; with CG = 2 a CTA PAIR computes a
//                       256 x 256 tile with one cta_group::2 MMA (each CTA stages its 128 P rows and
//                       HALF of the Q rows: 128 flop per shared-memory byte instead of 85, which is
//                       what the ~12 TB/s L2 -> SM path can feed at cuBLAS speed).
//   decode  (M <= 128): swapped: P = weights (vocab rows), Q = activations (BN = 32 / 64 / 128), so
//                       a batch of 32 runs 128 x 32 MMAs with no wasted rows and the kernel is a
//                       pure HBM stream over W (lm_head: 1.05 GB / step).
// Persistent CTAs (one per SM, or one pair per 2 SMs), warp roles:
//   warp 0   TMA producer (STAGES-deep ring, full / empty mbarriers)
//   warp 1   MMA issuer (leader CTA of a pair only); tcgen05.commit releases ring slots and
//            publishes the accumulator; owns the TMEM allocation
//   warps 2-5 epilogue: tcgen05.ld of the finished accumulator (double-buffered in TMEM, so the
//            MMAs of tile i+1 overlap the drain of tile i), bias, convert, vectorised stores
// Roofline: prefill = tensor (2*M*N*K flop); decode = HBM (N*K*2 bytes).
#include "dense_gemm_tc.cuh"

namespace b200 {
namespace dg {

template <bool OUT_F32>
static bool launch_out(const void* x, const void* w, void* c, const __half* bias, int M, int N, int K,
                       int mode, cudaStream_t st) {
  if (M <= 128) {             // decode shapes: weights stream once, tokens are accumulator columns
    if (M <= 32) return launch_cfg<32, 1, true, OUT_F32>(x, w, c, bias, M, N, K, st);
    if (M <= 64) return launch_cfg<64, 1, true, OUT_F32>(x, w, c, bias, M, N, K, st);
    return launch_cfg<128, 1, true, OUT_F32>(x, w, c, bias, M, N, K, st);
  }
  if (mode == 1) return launch_cfg<256, 1, false, OUT_F32>(x, w, c, bias, M, N, K, st);
  return launch_cfg<256, 2, false, OUT_F32>(x, w, c, bias, M, N, K, st);
}

}  // namespace dg

// mode: 1 = single-CTA tiles, 2 = CTA pairs (cta_group::2).  false: shape not supported here.
bool launch_dense_gemm_tc(const void* x, const void* w, void* c, const void* bias, int M, int N, int K,
                          int out_f32, int mode, cudaStream_t st) {
  if (K % dg::kBK != 0 || N % 8 != 0) return false;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(c)) & 15)
    return false;
  const __half* b = static_cast<const __half*>(bias);
  return out_f32 ? dg::launch_out<true>(x, w, c, b, M, N, K, mode, st)
                 : dg::launch_out<false>(x, w, c, b, M, N, K, mode, st);
}

// gate|up projection with the SiLU * mul epilogue: w rows interleaved in 128-blocks (gate, up, gate, ...),
// out [M, N/2] fp16.  false: shape not supported (the caller runs GEMM + silu_mul instead).
bool launch_dense_gemm_tc_silu(const void* x, const void* w, void* out, int M, int N, int K, int mode,
                               cudaStream_t st) {
  if (K % dg::kBK != 0 || N % 256 != 0 || M <= 128) return false;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(out)) & 15)
    return false;
  if (mode == 1) return dg::launch_cfg<256, 1, false, false, true>(x, w, out, nullptr, M, N, K, st);
  return dg::launch_cfg<256, 2, false, false, true>(x, w, out, nullptr, M, N, K, st);
}

// ---------------------------------------------------------------- W4 / W8 -> fp16 [N, K]
// One pass over a prepacked (tile-major) quantised weight: thread = output channel, it reads the
// 32 / 64 packed bytes of a 64-K chunk and writes the chunk's 128 bytes of fp16((q - z) * s) into
// row n of the K-major scratch -- the Q operand of the kernel above.  Same rounding as the
// register dequant of wna16_tc.cu (one rounding, on the scale multiply).
template <int BITS>
__global__ void __launch_bounds__(kTileN)
wna16_dequant_kernel(const uint32_t* __restrict__ bp, const __half* __restrict__ scales,
                     const uint32_t* __restrict__ qzeros, __half* __restrict__ out, int K, int N,
                     int group_size, int qfmt, int chunks_per_cta, int interleave) {
  const int nt = blockIdx.x, ch = threadIdx.x, n = nt * kTileN + ch;
  // interleave: the fused gate|up weight ([gate tiles | up tiles] along N) is written as
  // gate tile 0, up tile 0, gate tile 1, ... so a 256-row GEMM tile holds both halves of 128 channels
  const int half_tiles = gridDim.x >> 1;
  const int dst_tile = interleave ? (nt < half_tiles ? 2 * nt : 2 * (nt - half_tiles) + 1) : nt;
  const int n_dst = dst_tile * kTileN + ch;
  const int KC = K / kChunkK;
  const int c0 = blockIdx.y * chunks_per_cta, c1 = min(c0 + chunks_per_cta, KC);
  constexpr int W = 2 * BITS;                                  // packed words per thread per chunk
  constexpr int kWBytes = kTileN * kChunkK * BITS / 8;
  pdl_trigger();
  int cur_g = -1;
  DqConst dq = make_dq(__float2half(0.f), 0);
  for (int kc = c0; kc < c1; ++kc) {
    const uint8_t* src = reinterpret_cast<const uint8_t*>(bp) + (static_cast<size_t>(nt) * KC + kc) * kWBytes;
    uint32_t words[W];
#pragma unroll
    for (int sub = 0; sub < W / 4; ++sub) {
      const uint4 u = ld_nc_v4(src + sub * kTileN * 16 + ch * 16);
      words[sub * 4] = u.x; words[sub * 4 + 1] = u.y; words[sub * 4 + 2] = u.z; words[sub * 4 + 3] = u.w;
    }
    uint32_t o[32];
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      const int g = (kc * kChunkK + hf * 32) / group_size;
      if (g != cur_g) {
        cur_g = g;
        dq = make_dq(scales[static_cast<size_t>(g) * N + n], load_zero<BITS>(qzeros, qfmt, g, n, N));
      }
      if (BITS == 4) {
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          uint32_t o4[4];
          dequant4_word(words[hf * 4 + w], dq, o4);
#pragma unroll
          for (int e = 0; e < 4; ++e) o[hf * 16 + w * 4 + e] = o4[e];
        }
      } else {
#pragma unroll
        for (int w = 0; w < 8; ++w) {
          uint32_t o2[2];
          dequant8_word(words[(hf * 8 + w) % W], dq, o2);
          o[hf * 16 + w * 2] = o2[0];
          o[hf * 16 + w * 2 + 1] = o2[1];
        }
      }
    }
    uint4* dst = reinterpret_cast<uint4*>(out + static_cast<size_t>(n_dst) * K + kc * kChunkK);
#pragma unroll
    for (int e = 0; e < 8; ++e) dst[e] = make_uint4(o[e * 4], o[e * 4 + 1], o[e * 4 + 2], o[e * 4 + 3]);
  }
}

void launch_wna16_dequant(const uint32_t* bp, const __half* scales, const uint32_t* qzeros, __half* out,
                          int K, int N, int bits, int group_size, int qfmt, cudaStream_t st, int interleave) {
  const int KC = K / kChunkK;
  const int cpc = 8;
  dim3 grid(N / kTileN, (KC + cpc - 1) / cpc);
  if (bits == 4)
    wna16_dequant_kernel<4><<<grid, kTileN, 0, st>>>(bp, scales, qzeros, out, K, N, group_size, qfmt, cpc, interleave);
  else
    wna16_dequant_kernel<8><<<grid, kTileN, 0, st>>>(bp, scales, qzeros, out, K, N, group_size, qfmt, cpc, interleave);
  B200_CUDA_LAUNCH_CHECK();
}

}  // namespace b200

// Dequantise a prepacked W4 / W8 weight to fp16 [n, k] (row n = output channel, K-major).
extern "C" void b200_wna16_dequant_f16(const void* b_packed, const void* scales, const void* qzeros,
                                       void* out, int32_t k, int32_t n, int32_t bits, int32_t group_size,
                                       int32_t qfmt, int64_t stream) {
  using namespace b200;
  B200_CHECK_ARG(b_packed && scales && out, "wna16_dequant: null pointer");
  B200_CHECK_ARG((bits == 4 || bits == 8) && k % kChunkK == 0 && n % kTileN == 0, "wna16_dequant: bad shape");
  const int g = group_size <= 0 ? k : group_size;
  B200_CHECK_ARG(g % 32 == 0 && k % g == 0, "wna16_dequant: bad group size");
  launch_wna16_dequant(static_cast<const uint32_t*>(b_packed), static_cast<const __half*>(scales),
                       static_cast<const uint32_t*>(qzeros), static_cast<__half*>(out), k, n, bits, g, qfmt,
                       reinterpret_cast<cudaStream_t>(stream), 0);
}
