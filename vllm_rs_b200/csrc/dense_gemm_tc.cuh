// The dense tcgen05 GEMM of dense_gemm_tc.cu (which describes it) and dense_gated.cu.
#pragma once
#include <cstdlib>
#include <cstring>

#include "host/per_device.hpp"
#include "wna16.cuh"

namespace b200 {
namespace dg {

constexpr int kThreads = 192;
constexpr int kBM = 128;       // P rows per CTA = TMEM lanes
constexpr int kBK = 64;        // K elements per stage (one 128-byte swizzle row)
// P tiles per rasterisation group: a group's P panel (group_p * 128 * CG rows x K) stays in L2 while
// the Q panels stream past it once per group.  B200_DENSE_GROUP_P overrides (A/B testing).
static int group_p_env() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("B200_DENSE_GROUP_P");
    v = e ? atoi(e) : 0;
  }
  return v;
}

template <int BN, int CG>
struct Cfg {
  static constexpr int kPBytes = kBM * kBK * 2;                 // 16 KB
  static constexpr int kQRows = BN / CG;                        // Q rows staged by one CTA
  static constexpr int kQBytes = kQRows * kBK * 2;
  static constexpr int kStageBytes = kPBytes + kQBytes;
  static constexpr int kStages = (196 * 1024) / kStageBytes;    // 6 (pair, BN 256) / 4 / ... / 9 (BN 32)
  static constexpr int kBarOff = kStages * kStageBytes;
  static constexpr int kNumBars = 2 * kStages + 4;
  static constexpr int kTmemPtrOff = kBarOff + kNumBars * 8;
  static constexpr int kAlloc = kTmemPtrOff + 16 + 1024;
  static_assert(kStageBytes % 1024 == 0, "stage bases must stay 1024-byte aligned (SWIZZLE_128B)");
  static_assert(kAlloc <= 227 * 1024, "shared memory budget");
  static_assert(2 * BN <= 512, "two accumulators must fit TMEM");
};

struct Args {
  void* c;
  const __half* bias;
  int M, N;            // logical output [M, N], row stride N
  int p_rows, q_rows;  // rows of the P / Q operand (swap: N / M, else M / N)
  int KB;              // K / 64
  int tiles_p, tiles_q, group_p;
};

__device__ __forceinline__ void tile_coords(int t, const Args& a, int& p, int& q) {
  const int per_group = a.group_p * a.tiles_q;
  const int g = t / per_group, r = t - g * per_group;
  const int rows = min(a.group_p, a.tiles_p - g * a.group_p);
  q = r / rows;
  p = g * a.group_p + (r - q * rows);
}

// SILU (prefill gate|up projection, BN = 256, fp16 out): the weight rows arrive interleaved in blocks of
// 128 (gate channels [128t, 128t+128) then up channels of the same range, see wna16_dequant_kernel), so
// accumulator columns c and c + 128 of a tile are gate / up of ONE output channel and the epilogue
// writes silu(gate) * up straight into [M, N/2] (mlp.rs:451-469) -- no [M, N] round trip through HBM.
// GATED (bf16 operands, CTA pairs): gate rows and up rows of W stand one behind the other, a pair's first CTA stages 128 of the gate's and
// the second the up rows of the same channels; the epilogue activates the fp32 sums as they are and rounds once, to bf16.
template <int BN, int CG, bool SWAP, bool OUT_F32, bool SILU = false, bool GATED = false>
__global__ void __launch_bounds__(kThreads, 1)
dense_gemm_tc_kernel(const __grid_constant__ CUtensorMap pmap, const __grid_constant__ CUtensorMap qmap,
                     const Args a) {
  using C = Cfg<BN, CG>;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t rank = CG == 2 ? cluster_ctarank() : 0;
  const int unit = blockIdx.x / CG, nunits = gridDim.x / CG;      // a unit = a CTA or a CTA pair
  const int ntiles = a.tiles_p * a.tiles_q;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::kBarOff);
  uint64_t* empty = full + C::kStages;
  uint64_t* tfull = empty + C::kStages;        // [2] accumulator published
  uint64_t* tempty = tfull + 2;                // [2] accumulator drained (leader's copy is the one waited on)
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(smem + C::kTmemPtrOff);

  if (threadIdx.x == 0) {
    for (int i = 0; i < C::kStages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], 4 * CG);           // every epilogue warp of the unit
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    if (CG == 2) {
      tmem_alloc_cg2(tmem_ptr, 512);
      tmem_relinquish_cg2();
    } else {
      tmem_alloc(tmem_ptr, 512);
      tmem_relinquish();
    }
  }
  if (warp == 0 && lane == 0) {
    prefetch_tmap(&pmap);
    prefetch_tmap(&qmap);
  }
  tc_fence_before();
  __syncthreads();
  if (CG == 2) {          // the peer's barriers must be initialised before anything signals them
    cluster_arrive();
    cluster_wait();
  }
  tc_fence_after();
  pdl_trigger();
  pdl_wait();             // activations (and, after a dequant pass, the weights) come from earlier kernels
  const uint32_t tmem_base = *tmem_ptr;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (every CTA)
    if (elect_one()) {
      uint32_t kit = 0;
      for (int t = unit; t < ntiles; t += nunits) {
        int p, q;
        tile_coords(t, a, p, q);
        const int prow = (p * CG + static_cast<int>(rank)) * kBM;
        const int qrow = GATED ? static_cast<int>(rank) * (a.N >> 1) + q * C::kQRows : q * BN + static_cast<int>(rank) * C::kQRows;
        for (int kb = 0; kb < a.KB; ++kb, ++kit) {
          const int s = kit % C::kStages;
          mbar_wait_bounded(&empty[s], ((kit / C::kStages) & 1) ^ 1);
          uint8_t* pdst = smem + s * C::kStageBytes;
          uint8_t* qdst = pdst + C::kPBytes;
          if (CG == 1) {
            mbar_arrive_expect_tx(&full[s], C::kStageBytes);
            tma_load_2d(pdst, &pmap, &full[s], kb * kBK, prow);
            tma_load_2d(qdst, &qmap, &full[s], kb * kBK, qrow);
          } else {
            // both CTAs' bytes complete on the LEADER's barrier, which expects the pair's total
            if (rank == 0) mbar_arrive_expect_tx(&full[s], 2 * C::kStageBytes);
            const uint32_t lbar = mapa_shared(smem_u32(&full[s]), 0);
            tma_load_2d_cg2(pdst, &pmap, lbar, kb * kBK, prow);
            tma_load_2d_cg2(qdst, &qmap, lbar, kb * kBK, qrow);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader CTA)
    if (rank == 0 && elect_one()) {
      const uint32_t idesc = make_idesc_f16(kBM * CG, BN) | (GATED ? (1u << 7) | (1u << 10) : 0u);       // bf16 operands
      uint32_t kit = 0;
      int it = 0;
      for (int t = unit; t < ntiles; t += nunits, ++it) {
        const int buf = it & 1;
        mbar_wait_bounded(&tempty[buf], ((it >> 1) & 1) ^ 1);     // epilogue drained this accumulator
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + buf * BN;
        for (int kb = 0; kb < a.KB; ++kb, ++kit) {
          const int s = kit % C::kStages;
          mbar_wait_bounded(&full[s], (kit / C::kStages) & 1);
          tc_fence_after();
          const uint32_t pbase = smem_u32(smem + s * C::kStageBytes);
          const uint64_t adesc = make_smem_desc_sw128(pbase);
          const uint64_t bdesc = make_smem_desc_sw128(pbase + C::kPBytes);
#pragma unroll
          for (int ks = 0; ks < kBK / 16; ++ks) {
            const uint32_t acc = (kb > 0 || ks > 0) ? 1u : 0u;
            if (CG == 2)
              tc_mma_ss_cg2(d_tmem, adesc + static_cast<uint64_t>(ks * 2), bdesc + static_cast<uint64_t>(ks * 2),
                            idesc, acc);
            else
              tc_mma_ss(d_tmem, adesc + static_cast<uint64_t>(ks * 2), bdesc + static_cast<uint64_t>(ks * 2),
                        idesc, acc);
          }
          if (CG == 2) tc_commit_cg2(&empty[s], 3); else tc_commit(&empty[s]);
        }
        if (CG == 2) tc_commit_cg2(&tfull[buf], 3); else tc_commit(&tfull[buf]);
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue warps (every CTA)
    const int q4 = warp & 3;                          // TMEM lane quarter this warp may read
    const uint32_t lane_base = static_cast<uint32_t>(q4 * 32) << 16;
    int it = 0;
    for (int t = unit; t < ntiles; t += nunits, ++it) {
      int p, q;
      tile_coords(t, a, p, q);
      const int buf = it & 1;
      mbar_wait_bounded(&tfull[buf], (it >> 1) & 1);
      tc_fence_after();
      const int prow = (p * CG + static_cast<int>(rank)) * kBM + q4 * 32 + lane;    // this thread's P row
      if (GATED) {
        const int half_n = a.N >> 1;
#pragma unroll 1
        for (int c0 = 0; c0 < BN / 2; c0 += 32) {
          uint32_t g[32], u[32];
          tmem_ld_x32(tmem_base + lane_base + buf * BN + c0, g);
          tmem_ld_x32(tmem_base + lane_base + buf * BN + BN / 2 + c0, u);
          tc_wait_ld();
          const int col = q * (BN / 2) + c0;          // output channel of g[0]
          if (prow < a.M && col < half_n) {
            __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(a.c) + static_cast<size_t>(prow) * half_n + col;
            auto act = [&](int j) {
              const float x = __uint_as_float(g[j]);
              return x / (1.f + expf(-x)) * __uint_as_float(u[j]);
            };
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              uint32_t w[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) w[e] = pack16x2<true>(act(j + 2 * e), act(j + 2 * e + 1));
              if (col + j + 8 <= half_n) *reinterpret_cast<uint4*>(dst + j) = make_uint4(w[0], w[1], w[2], w[3]);
            }
          }
        }
      } else if (SILU) {
        const int half_n = a.N >> 1;
#pragma unroll 1
        for (int c0 = 0; c0 < BN / 2; c0 += 32) {
          uint32_t g[32], u[32];
          tmem_ld_x32(tmem_base + lane_base + buf * BN + c0, g);
          tmem_ld_x32(tmem_base + lane_base + buf * BN + BN / 2 + c0, u);
          tc_wait_ld();
          const int col = q * (BN / 2) + c0;          // output channel of g[0]
          if (prow < a.M && col < half_n) {
            __half* dst = reinterpret_cast<__half*>(a.c) + static_cast<size_t>(prow) * half_n + col;
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              uint32_t w[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                // the two GEMM outputs are rounded to fp16 first: the values the unfused pipeline sees
                const float2 gg = __half22float2(u32_as_h2(pack_half2(__uint_as_float(g[j + 2 * e]), __uint_as_float(g[j + 2 * e + 1]))));
                const float2 uu = __half22float2(u32_as_h2(pack_half2(__uint_as_float(u[j + 2 * e]), __uint_as_float(u[j + 2 * e + 1]))));
                w[e] = pack_half2(gg.x / (1.f + __expf(-gg.x)) * uu.x, gg.y / (1.f + __expf(-gg.y)) * uu.y);
              }
              if (col + j + 8 <= half_n) *reinterpret_cast<uint4*>(dst + j) = make_uint4(w[0], w[1], w[2], w[3]);
            }
          }
        }
      } else
#pragma unroll 1
      for (int c0 = 0; c0 < BN; c0 += 32) {
        uint32_t v[32];
        tmem_ld_x32(tmem_base + lane_base + buf * BN + c0, v);
        tc_wait_ld();
        const int qcol = q * BN + c0;                 // first Q row (= accumulator column) of this block
        if (!SWAP) {
          // thread = token row m, 32 consecutive output channels
          const int m = prow;
          if (m < a.M && qcol < a.N) {
            if (a.bias) {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (qcol + j < a.N) v[j] = __float_as_uint(__uint_as_float(v[j]) + __half2float(a.bias[qcol + j]));
            }
            if (OUT_F32) {
              float* dst = reinterpret_cast<float*>(a.c) + static_cast<size_t>(m) * a.N + qcol;
#pragma unroll
              for (int j = 0; j < 32; j += 4)
                if (qcol + j + 4 <= a.N)
                  *reinterpret_cast<uint4*>(dst + j) = make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]);
            } else {
              __half* dst = reinterpret_cast<__half*>(a.c) + static_cast<size_t>(m) * a.N + qcol;
#pragma unroll
              for (int j = 0; j < 32; j += 8)
                if (qcol + j + 8 <= a.N) {
                  uint4 o;
                  o.x = pack_half2(__uint_as_float(v[j]), __uint_as_float(v[j + 1]));
                  o.y = pack_half2(__uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
                  o.z = pack_half2(__uint_as_float(v[j + 4]), __uint_as_float(v[j + 5]));
                  o.w = pack_half2(__uint_as_float(v[j + 6]), __uint_as_float(v[j + 7]));
                  *reinterpret_cast<uint4*>(dst + j) = o;
                }
            }
          }
        } else {
          // thread = output channel n (a weight row), columns = tokens: a warp writes 32
          // consecutive channels of one token row per store
          const int n = prow;
          if (n < a.N) {
            const float bv = a.bias ? __half2float(a.bias[n]) : 0.f;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const int m = qcol + j;
              if (m < a.M) {
                const float x = __uint_as_float(v[j]) + bv;
                if (OUT_F32)
                  reinterpret_cast<float*>(a.c)[static_cast<size_t>(m) * a.N + n] = x;
                else
                  reinterpret_cast<__half*>(a.c)[static_cast<size_t>(m) * a.N + n] = __float2half_rn(x);
              }
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (CG == 2 && rank != 0)
          mbar_arrive_cluster(mapa_shared(smem_u32(&tempty[buf]), 0));
        else
          mbar_arrive(&tempty[buf]);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (CG == 2) {          // neither CTA may leave (or free TMEM) while its peer can still touch it
    cluster_arrive();
    cluster_wait();
  }
  if (warp == 1) {
    tc_fence_after();
    if (CG == 2) tmem_dealloc_cg2(tmem_base, 512); else tmem_dealloc(tmem_base, 512);
  }
}

static bool make_map(CUtensorMap* map, const void* base, int rows, int K, int box_rows, bool bf16 = false) {
  const uint64_t dims[2] = {static_cast<uint64_t>(K), static_cast<uint64_t>(rows)};
  const uint64_t strides[1] = {static_cast<uint64_t>(K) * 2};
  const uint32_t box[2] = {kBK, static_cast<uint32_t>(box_rows)};
  const uint32_t es[2] = {1, 1};
  return encode_tensor_map(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides,
                           box, es, CU_TENSOR_MAP_SWIZZLE_128B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B) == CUDA_SUCCESS;
}

template <int BN, int CG, bool SWAP, bool OUT_F32, bool SILU = false, bool GATED = false>
static bool launch_cfg(const void* x, const void* w, void* c, const __half* bias, int M, int N, int K,
                       cudaStream_t st) {
  using C = Cfg<BN, CG>;
  const void* pbase = SWAP ? w : x;
  const void* qbase = SWAP ? x : w;
  Args a;
  a.c = c; a.bias = bias; a.M = M; a.N = N;
  a.p_rows = SWAP ? N : M;
  a.q_rows = SWAP ? M : N;
  a.KB = K / kBK;
  a.tiles_p = (a.p_rows + kBM * CG - 1) / (kBM * CG);
  a.tiles_q = GATED ? (N / 2 + C::kQRows - 1) / C::kQRows : (a.q_rows + BN - 1) / BN;
  // 16 P tiles per group measured best on all four Llama-3-8B prefill shapes (M = 8192: 1390-1450 TF/s
  // with CTA pairs; 8 re-reads the weight panels from HBM 6x, 32 thrashes L2 at K = 14336)
  {
    int gp = 16;
    if (group_p_env() > 0) gp = group_p_env();
    a.group_p = gp;
  }
  CUtensorMap pmap, qmap;
  if (!make_map(&pmap, pbase, a.p_rows, K, kBM, GATED) || !make_map(&qmap, qbase, a.q_rows, K, C::kQRows, GATED)) {
    set_error(2, "dense_gemm_tc: cuTensorMapEncodeTiled failed");
    return true;
  }
  auto kern = dense_gemm_tc_kernel<BN, CG, SWAP, OUT_F32, SILU, GATED>;
  static OncePerDevice sized;
  int dev = 0;
  cudaGetDevice(&dev);
  const cudaError_t set = sized(dev, [&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kAlloc); });
  if (set != cudaSuccess) {
    set_error(2, cudaGetErrorString(set));
    return true;
  }
  static const int max_units = [&] {
    if (CG == 1) return sm_count();
    const int n = max_active_clusters(kern, dim3(sm_count()), dim3(kThreads), C::kAlloc, dim3(2, 1, 1));
    return n > 0 ? n : sm_count() / 2;
  }();
  const int ntiles = a.tiles_p * a.tiles_q;
  const int units = ntiles < max_units ? ntiles : max_units;
  const cudaError_t e = launch_pdl_cluster(kern, dim3(units * CG), dim3(kThreads), C::kAlloc, st,
                                           dim3(CG, 1, 1), pmap, qmap, a);
  if (e != cudaSuccess) set_error(2, cudaGetErrorString(e));
  B200_CUDA_LAUNCH_CHECK();
  return true;
}

}  // namespace dg
}  // namespace b200
