// The grouped matrix products of routed experts on tcgen05 tensor cores (bf16 operands, fp32 accumulation; moe.cu has the
// formulas, the buckets and the fp32 / odd-size forms).
//
// Persistent blocks, one per SM, walk tiles of 128 slots (rows of ONE expert's bucket) x BN weight rows.  Warp 0 fetches 64-wide
// K blocks of both operands by TMA, of the rows only as many 32-row boxes as the bucket has, a full tile as one
// box (the two products of the prompt below: 75 / 52 -> 71 / 51 us).  Warp 1 issues the products into
// one of two TMEM accumulators, warps 2-9 apply the activation and store, through shared memory so that rows leave in whole
// sectors, under the products of the next tile.  A gated tile holds BN / 2 gate and BN / 2 up rows of the same features side by
// side, so the activation needs no second pass.  Token rows are first gathered into bucket order by a copy of their own (in
// space that the second product's results take later): gathering inside the product took longer than the product, by TMA
// gathers of four rows (~90 cycles each) as by cp.async, whose blocks need a wait and a fence on their way to the tensor core
// (prompt of 4096 rows, 16 experts, first product: 183 us and 103-139 us).  Two blocks of a cluster may share a tile of 256 slots, each
// with its own rows and half of the weight rows in shared memory: two thirds of the reads (that prompt's products 71 / 52 -> 66 / 52 us).
// The launches of a call, but for the sum of the choices, depend on each other as programs, so that the next one's start lies under
// the last one's end.  Replayed as a graph, without pairs and dependent launches and with both: 40 rows 41.5 -> 33.8 us, 4096 rows 172 -> 158.5.
//
// Measured, mma.sync kernel -> here (whole public call): 4096 rows of 2048, 16 experts of 512, 4 chosen: 709 -> 183 us, 32 rows, device time,
// 67 -> 36; 4096 wide, 32 experts of 1024: 3000 rows 1903 -> 406 us, 32 rows, device time, 202 -> 159.  moe.cu says which products are
// long enough to come here.
// Bound: tensor cores where experts get hundreds of rows, HBM (every hit expert's weights once) where they get few; BN is 256
// where that gives every SM two tiles, else 128 where that gives three SMs in four one (below that the launches are the bound),
// else 64.  Whole calls with BN = 64 / 128 / 256, 2048 wide, 16 experts of 512: 2 rows 47.8 / 47.5 / 49.2 us (128 / 64 / 32 tiles
// in the first product), 8 rows 56.0 / 45.6 / 48.5 (256 / 128 / 64), 300 rows 69.6 / 52.6 / 63.0, 4096 rows 388 / 243 / 187;
// 4096 wide, 32 experts of 1024: 32 rows 198 / 142 / 150 us, 300 rows 295 / 185 / 177, 3000 rows 1027 / 573 / 405.
#include "../../include/b200_vllm.h"
#include <cmath>
#include "moe_tc.cuh"

namespace b200 {
using namespace seqmix;
namespace moetc {

constexpr int kM = 128, kK = 64, kBox = 32, kThreads = 320, kEpiWarps = 8, kMaxExperts = 1024;
constexpr int kABytes = kM * 128;
constexpr int kPitch = 80, kOutBytes = kEpiWarps * 32 * kPitch;      // a warp's 32 rows x 64 bytes on their way out
constexpr uint32_t kHiSw128 = (1024 >> 4) | (1u << 14) | (2u << 29);

template <int BN, int CG> struct Cfg {                          // CG: blocks that share a tile
  static constexpr int kWRows = BN / CG;                       // weight rows staged by a block
  static constexpr int kStage = kABytes + kWRows * 128;
  static constexpr int kStages = 192 * 1024 / kStage;          // 4 / 6 / 8 (pairs: 6)
  static constexpr int kOutOff = kStages * kStage;
  static constexpr int kBarOff = kOutOff + kOutBytes;
  static constexpr int kSmem = kBarOff + (2 * kStages + 5) * 8 + 16 + (kMaxExperts + 1) * 4 + 1024;
};

struct Args {
  void* out;
  const int32_t* off;
  int E, KB, N, ntiles_n;          // KB: K blocks; N: output features; ntiles_n: tiles along them
  b200_expert_act act;
  int* err;
};

template <int CG>
__device__ __forceinline__ void mma_ss(uint32_t lead, uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t acc) {
  if constexpr (CG == 1)
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\t"
        "setp.ne.b32 q, %0, 0;\n\tsetp.ne.b32 p, %6, 0;\n\t"
        "mov.b64 da, {%2, %5};\n\tmov.b64 db, {%3, %5};\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%1], da, db, %4, p;\n\t}\n" ::"r"(lead),
        "r"(d), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(kHiSw128), "r"(acc)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\t"
        "setp.ne.b32 q, %0, 0;\n\tsetp.ne.b32 p, %6, 0;\n\t"
        "mov.b64 da, {%2, %5};\n\tmov.b64 db, {%3, %5};\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%1], da, db, %4, p;\n\t}\n" ::"r"(lead),
        "r"(d), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(kHiSw128), "r"(acc)
        : "memory");
}
// on this barrier in the blocks of `mask` (one block: its own)
template <int CG>
__device__ __forceinline__ void commit(uint32_t lead, uint64_t* bar, uint16_t mask = 3) {
  if constexpr (CG == 1)
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %0, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%1];\n\t}\n" ::"r"(lead),
        "r"(smem_u32(bar))
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %0, 0;\n\t"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%1], %2;\n\t}\n" ::"r"(lead),
        "r"(smem_u32(bar)), "h"(mask)
        : "memory");
}

// ACT as in moe.cu: 0 plain product, fp32 out; 1 SiLU gate, 2 squared ReLU, 3 clamped gate, bf16 out.  Rows in bucket order.  After a wait has given up (*fail) all others return at once and the loops run out.
template <int ACT, int BN, int CG>
__global__ void __launch_bounds__(kThreads, 1)
grouped_linear_tc_kernel(const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap tilemap,
                         const __grid_constant__ CUtensorMap wmap, const Args a) {
  constexpr bool GATED = ACT == 1 || ACT == 3;
  constexpr int FN = GATED ? BN / 2 : BN;          // output features of a tile
  constexpr int TM = kM * CG;                      // rows of a tile
  using C = Cfg<BN, CG>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::kBarOff);
  uint64_t* empty = full + C::kStages;
  uint64_t* tfull = empty + C::kStages;            // [2] accumulator complete
  uint64_t* tempty = tfull + 2;                    // [2] accumulator stored
  uint64_t* drained = tempty + 2;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(drained + 1);
  volatile int* fail = reinterpret_cast<volatile int*>(tmem_ptr + 1);
  int* first = reinterpret_cast<int*>(tmem_ptr + 4);         // [E + 1] first row tile of every expert
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int rank = CG == 2 ? static_cast<int>(cluster_ctarank()) : 0, unit = blockIdx.x / CG, units = gridDim.x / CG;

  pdl_trigger();
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&tfull[s], 1); mbar_init(&tempty[s], kEpiWarps * CG); }
    mbar_init(drained, 1);
    *fail = 0;
    fence_barrier_init();
    prefetch_tmap(&amap);
    prefetch_tmap(&tilemap);
    prefetch_tmap(&wmap);
  }
  if (warp == 1) {
    if constexpr (CG == 2) {
      tmem_alloc_cg2(tmem_ptr, 2 * BN);
      tmem_relinquish_cg2();
    } else {
      tmem_alloc(tmem_ptr, 2 * BN);
      tmem_relinquish();
    }
  }
  pdl_wait();                                      // buckets and rows come from the kernels before, and results go where they read
  if (warp == 2) {                                 // row tiles before every expert: a scan over the buckets' sizes
    int before = 0;
    for (int e0 = 0; e0 < a.E; e0 += 32) {
      const int e = e0 + lane;
      const int mine = e < a.E ? (a.off[e + 1] - a.off[e] + TM - 1) / TM : 0;
      int inc = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
      }
      if (e < a.E) first[e] = before + inc - mine;
      before += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) first[a.E] = before;
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (CG == 2) {                         // the other block's barriers are there
    cluster_arrive();
    cluster_wait();
  }
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_ptr, 0);
  const int ntiles = first[a.E] * a.ntiles_n;
  // tile -> expert, first slot, rows, first feature
  struct Tile { int e, s0, rows, n0; };
  auto tile_at = [&](int t) {
    const int m = t / a.ntiles_n;
    int lo = 0, hi = a.E - 1;                      // the last expert whose first tile is <= m (empty ones share their successor's)
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (first[mid] <= m) lo = mid; else hi = mid - 1;
    }
    const int b = a.off[lo], k = m - first[lo];
    return Tile{lo, b + k * TM, min(TM, a.off[lo + 1] - b - k * TM), (t - m * a.ntiles_n) * FN};
  };

  if (warp == 0) {
    // ------------------------------------------------------------ operands
    int s = 0, armed = 0;
    uint32_t ph = 0;
    bool free_ = true;
    for (int t = unit; t < ntiles && free_; t += units) {
      const Tile w = tile_at(t);
      // the boxes of this block's rows, and of the tile; a pair's second block has the up rows, or the second half of the plain ones
      const int all = (w.rows + kBox - 1) / kBox, boxes = min(max(all - rank * (kM / kBox), 0), kM / kBox), s0 = w.s0 + rank * kM;
      const int wrow = w.e * (GATED ? 2 : 1) * a.N + w.n0 + rank * (GATED ? a.N : C::kWRows);
      for (int kb = 0; kb < a.KB; ++kb) {
        free_ = __all_sync(0xffffffffu, mbar_wait_limited(&empty[s], ph ^ 1, fail, a.err));
        if (!free_) break;                         // a stage that did not come free is not armed again
        uint8_t* ad = smem + s * C::kStage;
        uint8_t* wd = ad + kABytes;
        if (elect_one()) {
          if constexpr (CG == 2) {                 // both blocks' bytes count on the first one's barrier
            if (rank == 0) mbar_arrive_expect_tx(&full[s], all * (kBox * 128) + BN * 128);
            const uint32_t bar = mapa_shared(smem_u32(&full[s]), 0);
            tma_load_2d_cg2(wd, &wmap, bar, kb * kK, wrow);
            if (boxes == kM / kBox) tma_load_2d_cg2(ad, &tilemap, bar, kb * kK, s0);
            else
              for (int i = 0; i < boxes; ++i) tma_load_2d_cg2(ad + i * (kBox * 128), &amap, bar, kb * kK, s0 + i * kBox);
          } else {
            mbar_arrive_expect_tx(&full[s], boxes * (kBox * 128) + BN * 128);
            tma_load_2d(wd, &wmap, &full[s], kb * kK, wrow);
            if (GATED) tma_load_2d(wd + FN * 128, &wmap, &full[s], kb * kK, wrow + a.N);
            if (boxes == kM / kBox) tma_load_2d(ad, &tilemap, &full[s], kb * kK, s0);      // a copy costs its issue, whatever its size
            else
              for (int i = 0; i < boxes; ++i) tma_load_2d(ad + i * (kBox * 128), &amap, &full[s], kb * kK, s0 + i * kBox);
          }
        }
        ++armed;
        if (++s == C::kStages) { s = 0; ph ^= 1; }
      }
    }
    if (lane == 0 && rank == 0 && *fail)           // copies in flight land before the block ends (a pair's second waits for its first)
      for (int i = 0; i < C::kStages && i < armed; ++i)
        mbar_wait_limited(&full[i], ((armed - 1 - i) / C::kStages) & 1, nullptr, a.err);
    __syncwarp();
  } else if (warp == 1 && rank == 0) {
    // ------------------------------------------------------------ products
    constexpr uint32_t idesc = make_idesc_f16(TM, BN) | (1u << 7) | (1u << 10);        // bf16 operands
    const uint32_t lead = elect_one() ? 1u : 0u;
    const uint32_t base = (smem_u32(smem) >> 4) | (1u << 16);
    int s = 0, it = 0;
    uint32_t ph = 0;
    for (int t = unit; t < ntiles; t += units, ++it) {
      const int buf = it & 1;
      mbar_wait_limited(&tempty[buf], ((it >> 1) & 1) ^ 1, fail, a.err);
      tc_fence_after();
      const uint32_t d = tmem + buf * BN;
      for (int kb = 0; kb < a.KB; ++kb) {
        mbar_wait_limited(&full[s], ph, fail, a.err);
        tc_fence_after();
        const uint32_t a_lo = base + s * (C::kStage >> 4), b_lo = a_lo + (kABytes >> 4);
#pragma unroll
        for (int ks = 0; ks < kK / 16; ++ks) mma_ss<CG>(lead, d, a_lo + ks * 2, b_lo + ks * 2, idesc, (kb | ks) ? 1u : 0u);
        commit<CG>(lead, &empty[s]);
        if (++s == C::kStages) { s = 0; ph ^= 1; }
      }
      commit<CG>(lead, &tfull[buf]);
    }
    if (*fail) {                                   // products in flight end before TMEM is given back
      commit<CG>(lead, drained, 1);
      mbar_wait_limited(drained, 0, nullptr, a.err);
    }
    __syncwarp();
  } else if (warp > 1) {
    // ------------------------------------------------------------ activation and stores
    // A warp reads its quarter of the rows, every other 32 columns; four lanes then write 64 bytes of a row.
    const int q4 = warp & 3;
    const uint32_t lanes = static_cast<uint32_t>(q4 * 32) << 16;
    uint8_t* stage = smem + C::kOutOff + (warp - 2) * 32 * kPitch;
    const int sub = (lane & 3) * 16;
    int it = 0;
    for (int t = unit; t < ntiles; t += units, ++it) {
      const Tile w = tile_at(t);
      const int buf = it & 1;
      mbar_wait_limited(&tfull[buf], (it >> 1) & 1, fail, a.err);
      __syncwarp();
      tc_fence_after();
      const uint32_t src = tmem + lanes + buf * BN;
      const int rows = w.rows - rank * kM - q4 * 32;               // of this warp
      // the staged rows' bytes [b, b + 64) of a tile row whose first column is n0
      auto store = [&](int b, int elem) {
        __syncwarp();
        uint8_t* dst = static_cast<uint8_t*>(a.out) + (static_cast<size_t>(w.s0 + rank * kM + q4 * 32) * a.N + w.n0) * elem + b + sub;
        if (w.n0 * elem + b + sub < a.N * elem) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int rw = i * 8 + (lane >> 2);
            if (rw < rows)
              *reinterpret_cast<uint4*>(dst + static_cast<size_t>(rw) * a.N * elem) =
                  *reinterpret_cast<const uint4*>(stage + rw * kPitch + sub);
          }
        }
        __syncwarp();
      };
      if (rows > 0) {
#pragma unroll 1
        for (int c = warp < 6 ? 0 : 32; c < FN; c += 64) {
          uint32_t v[32], u[GATED ? 32 : 1];
          tmem_ld_x32(src + c, v);
          if constexpr (GATED) tmem_ld_x32(src + FN + c, u);
          tc_wait_ld();
          if constexpr (ACT == 0) {
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
#pragma unroll
              for (int i = 0; i < 16; i += 4)
                *reinterpret_cast<uint4*>(stage + lane * kPitch + i * 4) =
                    make_uint4(v[hf * 16 + i], v[hf * 16 + i + 1], v[hf * 16 + i + 2], v[hf * 16 + i + 3]);
              store((c + hf * 16) * 4, 4);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              float x = __uint_as_float(v[i]);
              if constexpr (GATED) {
                x = expert_gate<ACT>(x, __uint_as_float(u[i]), a.act);
              } else {
                x = fmaxf(x, 0.f);
                x *= x;
              }
              v[i] = __float_as_uint(x);
            }
#pragma unroll
            for (int i = 0; i < 32; i += 8)
              *reinterpret_cast<uint4*>(stage + lane * kPitch + i * 2) =
                  make_uint4(pack16x2<true>(__uint_as_float(v[i]), __uint_as_float(v[i + 1])),
                             pack16x2<true>(__uint_as_float(v[i + 2]), __uint_as_float(v[i + 3])),
                             pack16x2<true>(__uint_as_float(v[i + 4]), __uint_as_float(v[i + 5])),
                             pack16x2<true>(__uint_as_float(v[i + 6]), __uint_as_float(v[i + 7])));
            store(c * 2, 2);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        // (what the products overwrite has been read; a release at cluster scope would wait for the results' stores)
        if (CG == 2 && rank != 0)
          asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(mapa_shared(smem_u32(&tempty[buf]), 0)) : "memory");
        else
          mbar_arrive(&tempty[buf]);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (CG == 2) {                         // neither block goes while the other can reach its memory
    cluster_arrive();
    cluster_wait();
  }
  if (warp == 1) {
    tc_fence_after();
    if constexpr (CG == 2) tmem_dealloc_cg2(tmem, 2 * BN);
    else tmem_dealloc(tmem, 2 * BN);
  }
}

static bool map_2d(CUtensorMap* m, const void* base, uint64_t rows, int K, uint32_t box_rows) {
  const uint64_t dims[2] = {static_cast<uint64_t>(K), rows}, strides[1] = {static_cast<uint64_t>(K) * 2};
  const uint32_t box[2] = {kK, box_rows}, es[2] = {1, 1};
  return encode_tensor_map(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, es,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B) == CUDA_SUCCESS;
}

// a [pairs, K] in bucket order
template <int ACT, int BN, int CG = 1>
static void launch(void* out, const void* a, const void* w, const int32_t* off, int pairs, int E, int K, int N,
                   const b200_expert_act& act, cudaStream_t st) {
  constexpr bool GATED = ACT == 1 || ACT == 3;
  constexpr int FN = GATED ? BN / 2 : BN;
  Args g{out, off, E, (K + kK - 1) / kK, N, (N + FN - 1) / FN, act, wait_error_flag()};
  CUtensorMap amap, tilemap, wmap;
  const bool ok = map_2d(&amap, a, pairs, K, kBox) && map_2d(&tilemap, a, pairs, K, kM) &&
                  map_2d(&wmap, w, static_cast<uint64_t>(E) * (GATED ? 2 : 1) * N, K, CG == 2 ? BN / 2 : FN);
  if (!ok || !g.err) {
    set_error(2, "grouped_linear_tc: cuTensorMapEncodeTiled failed");
    return;
  }
  auto kern = grouped_linear_tc_kernel<ACT, BN, CG>;
  static OncePerDevice sized;
  if (!allow_smem(sized, kern, Cfg<BN, CG>::kSmem)) return;
  const int most = std::min(pairs, E + pairs / (kM * CG)) * g.ntiles_n;        // no step has more tiles
  const dim3 grid(std::min(most, sm_count() / CG) * CG);
  if constexpr (CG == 1) {
    launch_pdl(kern, grid, dim3(kThreads), Cfg<BN, CG>::kSmem, st, amap, tilemap, wmap, g);
  } else {
    const cudaError_t e = launch_pdl_cluster(kern, grid, dim3(kThreads), Cfg<BN, CG>::kSmem, st, dim3(CG), amap, tilemap, wmap, g);
    if (e != cudaSuccess) set_error(2, cudaGetErrorString(e));
  }
  B200_CUDA_LAUNCH_CHECK();
}

template <int ACT>
static void launch_bn(void* out, const void* a, const void* w, const int32_t* off, int pairs, int E, int K, int N,
                      const b200_expert_act& act, cudaStream_t st) {
  constexpr int G = ACT == 1 || ACT == 3 ? 2 : 1;
  const int row_tiles = std::max(std::min(E, pairs), pairs / kM);
  // Pairs of blocks where their tiles, twice as high, do not cost more turns: a pair's turn takes 0.8 - 0.9 of a block's (first product
  // of the prompt above 73 000 and 93 000 cycles for four, second 60 000 and 66 000 for eight).  Calls replayed
  // as a graph, single blocks and pairs, us: 16 experts of 512, 2048 wide, 2000 rows 95.4 and 99.1 (two turns and three), 2500 rows 121 and 116, 4096
  // rows 174 and 165, 8000 rows 302 and 299; 64 experts of 1024, 8 chosen, 2500 rows 363 and 338, 4096 rows 516 and 497.
  const auto turns = [&](int rows, int slots) {            // half a tile of every bucket is past its end
    const double tiles = std::max<double>(std::min(E, pairs), E * 0.5 + static_cast<double>(pairs) / rows) * ((N * G + 255) / 256);
    return std::ceil(tiles / slots);
  };
  if (row_tiles * ((N * G + 255) / 256) >= 2 * sm_count()) {
    // (buckets of fewer rows than a pair's tile leave its second block idle: 1000 rows, 8 of 64 experts, 218 single and 236)
    if (pairs >= 2 * kM * E && 0.85 * turns(2 * kM, sm_count() / 2) <= turns(kM, sm_count())) launch<ACT, 256, 2>(out, a, w, off, pairs, E, K, N, act, st);
    else launch<ACT, 256>(out, a, w, off, pairs, E, K, N, act, st);
  }
  else if (row_tiles * ((N * G + 127) / 128) >= sm_count() * 3 / 4) launch<ACT, 128>(out, a, w, off, pairs, E, K, N, act, st);
  else launch<ACT, 64>(out, a, w, off, pairs, E, K, N, act, st);
}

// out[slot] = h[pair_of_slot[slot] / top], rows of n16 16-byte pieces
__global__ void __launch_bounds__(256)
bucket_rows_kernel(uint4* __restrict__ out, const uint4* __restrict__ h, const int32_t* __restrict__ pair_of_slot, int pairs,
                   int top, int n16) {
  const int per = 256 / 32, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;       // a warp per row
  const int slot = blockIdx.x * per + warp;
  pdl_trigger();
  pdl_wait();
  if (slot >= pairs) return;
  const uint4* src = h + static_cast<size_t>(pair_of_slot[slot] / top) * n16;
  uint4* dst = out + static_cast<size_t>(slot) * n16;
  for (int i0 = lane; i0 < n16; i0 += 128) {
    uint4 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (i0 + 32 * i < n16) v[i] = __ldg(src + i0 + 32 * i);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (i0 + 32 * i < n16) dst[i0 + 32 * i] = v[i];
  }
}

}  // namespace moetc

bool grouped_linear_tc(int act_kind, void* out, const void* a, const void* w, const int32_t* off, const int32_t* pair_of_slot,
                       void* rows, int pairs, int top, int E, int K, int N, const b200_expert_act& act, cudaStream_t st) {
  using namespace moetc;
  const uintptr_t ptrs = reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w) |
                         reinterpret_cast<uintptr_t>(rows);
  if (K % 8 != 0 || N % 8 != 0 || E > kMaxExperts || (ptrs & 15) || (act_kind != 0 && !rows)) return false;
  if (act_kind != 0) {
    launch_pdl(bucket_rows_kernel, dim3((pairs + 7) / 8), dim3(256), 0, st, static_cast<uint4*>(rows), static_cast<const uint4*>(a),
               pair_of_slot, pairs, top, K / 8);
    B200_CUDA_LAUNCH_CHECK();
    a = rows;
  }
  switch (act_kind) {
    case 0: launch_bn<0>(out, a, w, off, pairs, E, K, N, act, st); break;
    case 1: launch_bn<1>(out, a, w, off, pairs, E, K, N, act, st); break;
    case 2: launch_bn<2>(out, a, w, off, pairs, E, K, N, act, st); break;
    default: launch_bn<3>(out, a, w, off, pairs, E, K, N, act, st); break;
  }
  return true;
}

}  // namespace b200
