// W4A16 / W8A16 GEMM on tcgen05 for decode batches: units of 128 channels x 128 K cut evenly over the SMs.
//
// The reference's arithmetic: weights (q - z) * s rounded once to fp16, fp32 sums.
//
// What bounds it.  A unit of 4-bit weights is 356 SM cycles of HBM (8 KB at 6.5 TB/s over 148 SMs) and 256 of the fp16 pipe, which takes two
// cycles for each of the eight instructions that turn a packed word of a warp into weights; the loop below without its barriers
// runs at 305.  Beside them every barrier is latency: a wait that passes takes 165 cycles, so one block's four groups and two
// issuers ask early (test_wait) for what they need next, and a unit is as large as tensor memory allows.  It runs at about 450 per unit
// (4-bit, 32 tokens; 530 with 64); 8-bit units at 740, which is HBM.  The rest is fixed time per launch, some 3 us: the previous
// kernel's end, the activations' way to shared memory (1300 cycles beside the weights' copies), the meeting of a tile's parts, and code that
// runs once, as fast as it is fetched (so the finalisers are short loops; SiLU's division takes 0.4 of
// 20.8 us at 4096 x 28672).
//
// Layout.  Sixteen warps dequantise: four groups take the block's units in turn, a warp has 32 channels (its quarter of the tensor memory's
// lanes) and writes 128 K of them as the A operand; the activations, by TMA, are the B operand.  Even and odd units have an issuer and an
// accumulator each.  Weights never wait for the previous kernel; scales and zero points are asked for two units ahead.  With
// SiLU a tile is 64 gate channels and their 64 up channels, so that every epilogue finds its operands in one tile.
//
// Meetings.  Parts of one size meet in a cluster: every block sends the others their rows' sums by bulk copies and finalises its own rows
// (through the L2: 4000 cycles more).  Ranges cut anywhere write the part of a tile that others share to the workspace; the last to
// arrive, by an atomic that also resets itself, sums in the order of K.  A block whose last tile has already been visited by
// all others keeps its part.
//
// us at 32 tokens, here and in wna16_tc_dec.cu: 4096 x 6144 7.2 / 8.8, 4096 x 4096 6.4 / 7.4, 4096 x 28672 19.5 / 30.2, 14336 x 4096 12.0 / 13.6,
// 2048 x 2560 4.9 / 6.4, 5632 x 2048 5.6 / 6.7, 8192 x 10240 16.9 / 21.2, 8192 x 57344 63 / 96, 28672 x 8192 33.4 / 42.7.
#include <atomic>
#include <cstring>

#include "host/per_device.hpp"
#include "host/unit_cut.hpp"
#include "wna16.cuh"

namespace b200 {
namespace ts {

constexpr int kUnitK = 128;
constexpr int kGroups = 4;                     // dequantising groups: four warps, the 128 channels of a unit
constexpr int kDqWarps = 4 * kGroups;
constexpr int kDqThreads = kDqWarps * 32;
constexpr int kWWarp = kDqWarps, kXWarp = kWWarp + 1, kMmaWarp = kXWarp + 1;      // two of the last
constexpr int kThreads = (kMmaWarp + 2) * 32;  // 20 warps leave 96 registers
constexpr int kPlaces = 6;                     // of dequantised units in tensor memory, 64 columns each

template <int BITS, int NT>
struct Cfg {
  static constexpr int kWBytes = kTileN * kUnitK * BITS / 8;
  static constexpr int kXBox = NT * 128, kXBytes = 2 * kXBox;      // two boxes of 64 K, 128-byte swizzle
  static constexpr int kSumBytes = NT * kTileN * 4;                 // the block's sums
  static constexpr int kTakeBytes = (NT == 16 ? 18 : NT) * kTileN * 4;      // its rows' sums of up to seven other blocks
  // Places of two units each.  Activations come 1300 cycles after they are asked for, beside the weights' copies.  The weights' places
  // are an even number: a place then always belongs to the same two groups, of which each has seen its last use when it asks for
  // the next (copies do not end in order, and a barrier two phases behind looks like one that is ready).
  static constexpr int kXPairs = NT == 16 ? 8 : NT == 32 ? (BITS == 4 ? 5 : 4) : 3;
  static constexpr int kFit = (225 * 1024 - kXPairs * 2 * kXBytes - kSumBytes - kTakeBytes) / (4 * kWBytes) * 2;
  static constexpr int kWPairs = kFit < 8 ? kFit : 8;
  static constexpr int kXOff = 0, kWOff = kXPairs * 2 * kXBytes, kSumOff = kWOff + kWPairs * 2 * kWBytes;
  static constexpr int kTakeOff = kSumOff + kSumBytes, kAlloc = kTakeOff + kTakeBytes + 1024;         // the start is aligned to 1024 bytes
  static constexpr int kDCols = NT < 32 ? 32 : NT;                  // an accumulator for even units, one for odd ones
  static constexpr int kACol = 2 * kDCols;
  static_assert(kACol + kPlaces * 64 <= 512 && kWPairs >= 2 && kAlloc <= 226 * 1024, "budgets");
};

struct Args {
  const uint8_t* bp;
  const __half* scales;
  const uint32_t* qzeros;
  int* err;              // set by a wait that gave up
  int M, K, N, qfmt;
  int gshift;            // log2(group_size / 128); 30: one group
  int U;                 // units per tile
  int cluster;           // blocks of a tile that meet in shared memory; 0: ranges cut anywhere
  int rows;              // finalised by each block of a cluster
  UnitCut cut;
  UnitDiv by_U;
  SplitOut o;
};

template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t at, uint32_t (&v)[N]) {
  static_assert(N == 4 || N == 8 || N == 16, "columns");
  if constexpr (N == 16) {
    tmem_ld_x16(at, v);
  } else if constexpr (N == 8) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(at)
                 : "memory");
  } else {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                 : "r"(at)
                 : "memory");
  }
}
__device__ __forceinline__ void tmem_st_x32(uint32_t at, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(at),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
      "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
      "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]),
      "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
      : "memory");
}
__device__ __forceinline__ void arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// A wait that gives up after some 2^24 polls (or when another one of the block has) and says so.
__device__ __forceinline__ bool wait(uint32_t bar, uint32_t parity, volatile int* fail, int* err) {
#pragma unroll 1
  for (int i = 0; !mbar_try_wait_addr(bar, parity); ++i)
    if (*fail || i > (1 << 24)) {
      *fail = 1;
      *reinterpret_cast<volatile int*>(err) = 1;
      return false;
    }
  return true;
}
// The same for a whole warp, whose lanes go on together: what follows (tcgen05 instructions, barriers) asks for all of them at once.
__device__ __forceinline__ void wait_warp(uint32_t bar, uint32_t parity, volatile int* fail, int* err) {
  wait(bar, parity, fail, err);
  __syncwarp();
}
// Asked early, looked at later: whether a wait would pass.
__device__ __forceinline__ void wait_probed(uint32_t ok, uint32_t bar, uint32_t parity, volatile int* fail, int* err) {
  if (!__all_sync(0xffffffffu, ok)) wait_warp(bar, parity, fail, err);
}
// A place of a ring of n and the parity of its use.
struct Ring {
  int s;
  uint32_t ph;
  __device__ __forceinline__ void next(int step, int n) {
    s += step;
    if (s >= n) {
      s -= n;
      ph ^= 1;
    }
  }
};


constexpr int kNone = -1;
// An arrival that hands nothing over (a release waits for the block's stores: some 700 cycles).
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
// From this block's shared memory to another one's; the bytes count on that one's barrier.
__device__ __forceinline__ void send_cluster(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "r"(src),
               "r"(bytes), "r"(bar)
               : "memory");
}
// A row's sums (a1: of the partner channels) finalised by a warp; with SiLU, where 64 gate channels and their 64 up channels make a tile, two
// rows, `first` and the next.
template <int EPI>
__device__ __forceinline__ void finish_row(const SplitOut& o, int tile, int lane, int first, int end, const float (&a0)[4],
                                           const float (&a1)[4]) {
  constexpr bool kSilu = EPI == B200_EPI_SILU_MUL;
  const FusedEpi& fe = o.fe;
  const int m = kSilu ? first + (lane >> 4) : first;
  const int n0 = kSilu ? tile * (kTileN / 2) + (lane & 15) * 4 : tile * kTileN + lane * 4;
  const EpiCol col = epi_col_at<EPI>(o, n0, kSilu ? n0 + (o.N >> 1) : EPI == kEpiRopeKv ? rope_partner(fe, n0) : -1);
  EpiRow er;
  epi_row_prefetch<EPI>(o, col, m, m < end, er);
  epi_row_prefetch2<EPI>(o, col, m < end, er);
  float scale = 1.f;
  if (fe.ssq_in) {
    float sum = warp_sum(ssq_lane_partial(fe.ssq_in + first * kSsqStride, fe.ssq_tiles, lane));
    if (kSilu) {
      const float other = warp_sum(first + 1 < end ? ssq_lane_partial(fe.ssq_in + (first + 1) * kSsqStride, fe.ssq_tiles, lane) : 0.f);
      if (lane >= 16) sum = other;
    }
    scale = rsqrtf(sum * fe.inv_dim + fe.eps);
  }
  epi_row_finish<EPI>(o, col, m, m < end, a0, a1, er, lane, scale);
}
__device__ __forceinline__ void add4(float (&a)[4], const float4& v) {
  a[0] += v.x;
  a[1] += v.y;
  a[2] += v.z;
  a[3] += v.w;
}
// Sums rows 0 .. M - 1 of a tile over its parts in the order of K and finalises them: sixteen warps, a row per warp (with SiLU two) at a
// time, P parts on their way.  The part of the block `own` (kNone: of no block) lies in `sums`, the others where part_of(block) says.
template <int EPI, class PartOf>
__device__ __forceinline__ void finish_tile(const SplitOut& o, int tile, int warp, int lane, int b0, int b1, int own,
                                            const float* sums, PartOf part_of) {
  constexpr bool kSilu = EPI == B200_EPI_SILU_MUL, kPair = kSilu || EPI == kEpiRopeKv;
  constexpr int P = 2, kRows = kSilu ? 2 : 1;
  const int c = kSilu ? (lane & 15) * 4 : lane * 4;
  const int n1 = EPI == kEpiRopeKv ? rope_partner(o.fe, tile * kTileN + c) : 0;
  const int pc = kSilu ? c + kTileN / 2 : n1 <= 0 ? 0 : n1 - tile * kTileN;
#pragma unroll 1
  for (int first = warp * kRows; first < o.M; first += kDqWarps * kRows) {
    const int m = kSilu ? min(first + (lane >> 4), o.M - 1) : first;
    float a0[4] = {0.f, 0.f, 0.f, 0.f}, a1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
    for (int b = b0; b <= b1; b += P) {
      float4 v0[P], v1[P];
#pragma unroll
      for (int i = 0; i < P; ++i) {
        const int bi = min(b + i, b1);
        const float* row = (bi == own ? sums : part_of(bi)) + m * kTileN;
        v0[i] = bi == own ? *reinterpret_cast<const float4*>(row + c) : __ldcg(reinterpret_cast<const float4*>(row + c));
        if (kPair) v1[i] = bi == own ? *reinterpret_cast<const float4*>(row + pc) : __ldcg(reinterpret_cast<const float4*>(row + pc));
      }
#pragma unroll
      for (int i = 0; i < P; ++i)
        if (b + i <= b1) {
          add4(a0, v0[i]);
          if (kPair) add4(a1, v1[i]);
        }
    }
    finish_row<EPI>(o, tile, lane, first, o.M, a0, a1);
  }
  if (EPI == kEpiPushPeers) push_signal(o.fe, warp * 32 + lane, kDqThreads, 2);
}

template <int BITS, int NT, int EPI>
__global__ void __launch_bounds__(kThreads, 1)
wna16_ts_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap, const __grid_constant__ Args a) {
  using C = Cfg<BITS, NT>;
  constexpr int SP = C::kWPairs, XP = C::kXPairs;
  constexpr bool kSilu = EPI == B200_EPI_SILU_MUL, kPairs = kSilu || EPI == kEpiRopeKv;
  extern __shared__ uint8_t smem_raw[];
  constexpr int kBars = 2 * SP + 2 * XP + 2 * kPlaces + 8;
  __shared__ uint64_t s_bars[kBars];
  uint64_t *const s_wfull = s_bars, *const s_wempty = s_wfull + SP, *const s_xfull = s_wempty + SP, *const s_xempty = s_xfull + XP,
                  *const s_stored = s_xempty + XP, *const s_free = s_stored + kPlaces, *const s_done = s_free + kPlaces,
                  *const s_flush = s_done + 2, *const s_taken = s_flush + 2, *const s_drained = s_taken + 1, *const s_written = s_drained + 2;
  __shared__ uint32_t s_tmem;
  __shared__ int s_last, s_first_last, s_alone, s_fail;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int U = a.U, N = a.N, M = a.M;
  const int u0 = a.cut.start(blockIdx.x), n = a.cut.start(blockIdx.x + 1) - u0;
  const int first_tile = a.by_U(u0), last_tile = a.by_U(u0 + n - 1);
  // tiles with other contributors than this block: the first, if another one follows, and the last
  const bool share_first = !a.cluster && first_tile < last_tile && u0 > first_tile * U;
  const bool share_last = !a.cluster && (u0 > last_tile * U || u0 + n < (last_tile + 1) * U);
  uint8_t* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  const uint32_t x_at = smem_u32(smem) + C::kXOff, w_at = smem_u32(smem) + C::kWOff;
  float* sums = reinterpret_cast<float*>(smem + C::kSumOff);
  pdl_trigger();
  if (threadIdx.x < kBars) {
    uint64_t* bar = s_bars + threadIdx.x;
    const int of = bar >= s_drained ? kDqWarps                 // its warps have read, or written, a tile's sums
                 : bar >= s_wempty && bar < s_xfull ? 8        // four warps for each of two units
                 : bar >= s_xempty && bar < s_stored ? 2       // the products of two units
                 : bar >= s_stored && bar < s_free ? 4 : 1;
    mbar_init(bar, of);
    fence_barrier_init();
  }
  if (threadIdx.x == 0) s_fail = s_last = s_first_last = s_alone = 0;
  __syncthreads();
  // (waited for before anything is sent to the other blocks, which have to be there)
  if (a.cluster) cluster_arrive_relaxed();

  if (warp == kWWarp) {
    // ------------------------------------------------------------ weights: they never wait for the previous kernel
    auto others = [&](int ct) { return static_cast<unsigned>(a.cut.block_of(ct * U + U - 1) - a.cut.block_of(ct * U)); };
    // The meeting of a tile's blocks: releases this one's part (`written` before) and acquires the others'.
    auto meet = [&](int ct) {
      unsigned old;
      asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(a.o.counters + ct) : "memory");
      const bool last = old == others(ct);
      if (last) a.o.counters[ct] = 0;                      // at rest again for the next launch
      return last ? 1 : 0;
    };
    if (elect_one()) {
      bool to_meet = share_first;
      Ring r{0, 1};
      int tile = first_tile, u = u0 - first_tile * U, i = 0;
      auto halves = [&](uint8_t* dst, uint64_t* bar) {
        // 64 gate channels, then 64 up channels: half tiles of [K / 32 or 16][128 channels x 16 bytes]
        const int sub = u * (kUnitK * BITS / 128);
        tma_load_4d(dst, &wmap, bar, 0, tile & 1, sub, tile >> 1);
        tma_load_4d(dst + C::kWBytes / 2, &wmap, bar, 0, tile & 1, sub, (N / kTileN / 2) + (tile >> 1));
        if (++u == U) {
          u = 0;
          ++tile;
        }
      };
#pragma unroll 1
      for (; i < n; i += 2) {
        if (!wait(smem_u32(&s_wempty[r.s]), r.ph, &s_fail, a.err)) break;
        const int units = min(2, n - i);
        uint64_t* bar = &s_wfull[r.s];
        mbar_arrive_expect_tx(bar, units * C::kWBytes);
        uint8_t* dst = smem + C::kWOff + r.s * (2 * C::kWBytes);
        if (kSilu) {
          halves(dst, bar);
          if (units > 1) halves(dst + C::kWBytes, bar);
        } else {
          bulk_load_1d(dst, a.bp + static_cast<size_t>(u0 + i) * C::kWBytes, units * C::kWBytes, bar);
        }
        r.next(1, SP);
        // the first tile's part is written some time after its last weights' place is filled again (the place is far ahead)
        if (to_meet && mbar_probe_addr(smem_u32(s_written), 0)) {
          s_first_last = meet(first_tile);
          to_meet = false;
        }
      }
      if (share_first || share_last) pdl_wait();
      if (to_meet) {
        wait(smem_u32(s_written), 0, &s_fail, a.err);
        s_first_last = meet(first_tile);
      }
      if (share_last && a.cut.whole) {
        // the last weights are on their way: if the others have all been here, nothing has to be written (parts of one size end together)
        unsigned seen;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.o.counters + last_tile) : "memory");
        s_alone = seen == others(last_tile);
        if (s_alone) a.o.counters[last_tile] = 0;
      }
      if (*reinterpret_cast<volatile int*>(&s_fail))       // copies in flight land before the block ends
        for (int j = max(0, i / 2 - SP); j < i / 2; ++j) mbar_wait_limited(&s_wfull[j % SP], (j / SP) & 1, nullptr, a.err);
    }
    __syncwarp();
    if (share_first || share_last) {
      if (a.cut.whole) asm volatile("bar.arrive 3, %0;" ::"n"(kDqThreads + 32) : "memory");
      if (share_last && !s_alone && elect_one()) {
        wait(smem_u32(s_written), share_first ? 1 : 0, &s_fail, a.err);
        s_last = meet(last_tile);
      }
      __syncwarp();
      asm volatile("bar.arrive 4, %0;" ::"n"(kDqThreads + 32) : "memory");
    }
  } else if (warp == kXWarp) {
    // ------------------------------------------------------------ activations (rows from M on come as zeros)
    if (elect_one()) {
      prefetch_tmap(&xmap);
      pdl_wait();
      Ring r{0, 1};
      int u = u0 - first_tile * U, i = 0;
#pragma unroll 1
      for (; i < n; i += 2) {
        if (!wait(smem_u32(&s_xempty[r.s]), r.ph, &s_fail, a.err)) break;
        const int units = min(2, n - i);
        mbar_arrive_expect_tx(&s_xfull[r.s], units * C::kXBytes);
        uint8_t* dst = smem + C::kXOff + r.s * (2 * C::kXBytes);
        tma_load_3d(dst, &xmap, &s_xfull[r.s], 0, 0, u * 2);
        if (++u == U) u = 0;
        if (units > 1) {
          tma_load_3d(dst + C::kXBytes, &xmap, &s_xfull[r.s], 0, 0, u * 2);
          if (++u == U) u = 0;
        }
        r.next(1, XP);
      }
      if (*reinterpret_cast<volatile int*>(&s_fail))
        for (int j = max(0, i / 2 - XP); j < i / 2; ++j) mbar_wait_limited(&s_xfull[j % XP], (j / XP) & 1, nullptr, a.err);
    }
  } else {
    if (warp == kMmaWarp) {
      tmem_alloc(&s_tmem, 512);
      tmem_relinquish();
    }
    tc_fence_before();
    named_bar_sync(1, kDqThreads + 64);
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    if (warp >= kMmaWarp) {
      // ------------------------------------------------------------ products of the even, or odd, units
      const int h = warp - kMmaWarp;
      if (elect_one()) {
        constexpr uint32_t idesc = make_idesc_f16(128, NT);
        const uint32_t d = tmem + h * C::kDCols;
        Ring p{h, 0}, x{0, 0};
        int i = h, turns = 0;                              // tiles in which this issuer had units
        const uint32_t xfull_at = smem_u32(s_xfull), stored_at = smem_u32(s_stored);
        uint32_t x_ok = 0, s_ok = 0;
#pragma unroll 1
        for (int ct = first_tile; ct <= last_tile; ++ct) {
          const int end = min((ct + 1) * U - u0, n);
          // Its own accumulator has been read.  A barrier for both issuers would not do: where a tile has one unit, the other issuer and the
          // readers end it alone, and a phase that this one has not looked at is followed by another of the same parity.
          if (turns > 0 && i < end) wait(smem_u32(&s_drained[h]), (turns - 1) & 1, &s_fail, a.err);
          uint32_t acc = 0;
#pragma unroll 1
          for (; i < end; i += 2) {
            if (!x_ok) wait(xfull_at + x.s * 8, x.ph, &s_fail, a.err);
            if (!s_ok) wait(stored_at + p.s * 8, p.ph, &s_fail, a.err);
            tc_fence_after();
            const uint32_t at = tmem + C::kACol + p.s * 64;
            const uint64_t b = make_smem_desc_sw128(x_at + (2 * x.s + h) * C::kXBytes);
            uint64_t* const free_ = &s_free[p.s];
            uint64_t* const empty = &s_xempty[x.s];
            p.next(2, kPlaces);
            x.next(1, XP);
            // A wait that passes costs 165 cycles, eight products 128: the next unit's are asked for under this one's products.
            s_ok = mbar_probe_addr(stored_at + p.s * 8, p.ph);
            x_ok = mbar_probe_addr(xfull_at + x.s * 8, x.ph);
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {
              tc_mma_ts(d, at + ks * 8, b + static_cast<uint64_t>((ks & 3) * 2 + (ks >> 2) * (C::kXBox >> 4)), idesc, acc);
              acc = 1;
            }
            tc_commit(free_);
            tc_commit(empty);
          }
          if (acc) {
            tc_commit(&s_done[h]);
            ++turns;
          }
        }
        if (*reinterpret_cast<volatile int*>(&s_fail)) {   // products in flight end before their memory is given back
          tc_commit(&s_flush[h]);
          mbar_wait_limited(&s_flush[h], 0, nullptr, a.err);
        }
      }
    } else {
      // ------------------------------------------------------------ dequantisation
      const int grp = warp >> 2, q4 = warp & 3, ch = q4 * 32 + lane;
      const uint32_t lanes = static_cast<uint32_t>(q4 * 32) << 16;
      constexpr int W = kUnitK * BITS / 32;              // words of a channel in a unit: 16 / 32
      constexpr int kSub = kSilu ? kTileN * 8 : kTileN * 16;
      const uint32_t q_at = w_at + (grp & 1) * C::kWBytes + (kSilu ? (ch >> 6) * (C::kWBytes / 2) + (ch & 63) * 16 : ch * 16);
      const int zshift = BITS == 8 ? 8 * (ch & 3) : a.qfmt == B200_QFMT_AWQ ? 4 * awq_nibble_of(ch & 7) : 4 * (ch & 7);
      const uint32_t zadd = (a.qfmt == B200_QFMT_AWQ && BITS == 4) ? 0 : 1;
      const bool has_z = a.qzeros != nullptr;
      // scale and zero point, asked for two units of the group ahead: (st, su) is the unit to be asked for next
      struct Sz {
        unsigned short s;
        uint32_t z;
      };
      int st = first_tile, su = u0 + grp - first_tile * U, s_col, z_col;
      auto columns = [&] {
        s_col = kSilu ? (st << 6) + (ch & 63) + (ch >> 6) * (N >> 1) : st * kTileN + ch;
        z_col = s_col / (32 / BITS);
      };
      columns();
      auto ask = [&] {
        if (su >= U) {
          do {
            su -= U;
            ++st;
          } while (su >= U);
          st = min(st, last_tile);                       // (past the block's units: nothing that is used)
          columns();
        }
        const int g = su >> a.gshift;
        su += kGroups;
        Sz v;
        v.s = __ldg(reinterpret_cast<const unsigned short*>(a.scales) + (g * N + s_col));
        v.z = has_z ? __ldg(a.qzeros + (g * (N * BITS / 32) + z_col)) : 0u;
        return v;
      };
      uint32_t q[W];
      Ring r{grp >> 1, 0}, p{grp, 1};
      const uint32_t s_wfull_at = smem_u32(s_wfull), s_wempty_at = smem_u32(s_wempty), s_free_at = smem_u32(s_free),
                     s_stored_at = smem_u32(s_stored);
      auto load = [&] {
        const uint32_t at = q_at + r.s * (2 * C::kWBytes);
#pragma unroll
        for (int sub = 0; sub < W / 4; ++sub)
          asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                       : "=r"(q[sub * 4]), "=r"(q[sub * 4 + 1]), "=r"(q[sub * 4 + 2]), "=r"(q[sub * 4 + 3])
                       : "r"(at + sub * kSub));
      };
      Sz sz0 = ask(), sz1 = ask();
      int i = grp, used[2] = {0, 0};
      bool waited = false, loaded = false;
#pragma unroll 1
      for (int ct = first_tile; ct <= last_tile; ++ct) {
        const int begin = max(ct * U - u0, 0), end = min((ct + 1) * U - u0, n);
#pragma unroll 1
        for (; i < end; i += kGroups) {
          if (!loaded) {
            wait_warp(s_wfull_at + r.s * 8, r.ph, &s_fail, a.err);
            load();
          }
          const uint32_t free_ = mbar_probe_addr(s_free_at + p.s * 8, p.ph);
          DqConst dq;
          {
            const uint32_t z = has_z ? ((sz0.z >> zshift) & ((1u << BITS) - 1)) + zadd : 1u << (BITS - 1);
            dq.s2 = u32_as_h2(static_cast<uint32_t>(sz0.s) * 0x00010001u);
            dq.zlo = u32_as_h2((0x6400u + z) * 0x00010001u);
            dq.zhi = u32_as_h2((0x5400u + (z << 4)) * 0x00010001u);
            sz0 = sz1;
            sz1 = ask();
          }
          const uint32_t at = tmem + C::kACol + p.s * 64 + lanes;
          auto dequant = [&](int hf, uint32_t (&v)[32]) {
            if constexpr (BITS == 4) {
#pragma unroll
              for (int w = 0; w < 8; ++w) {
                uint32_t o4[4];
                dequant4_word(q[hf * 8 + w], dq, o4);
#pragma unroll
                for (int e = 0; e < 4; ++e) v[w * 4 + e] = o4[e];
              }
            } else {
#pragma unroll
              for (int w = 0; w < 16; ++w) {
                uint32_t o2[2];
                dequant8_word(q[(hf * 16 + w) % W], dq, o2);
                v[w * 2] = o2[0];
                v[w * 2 + 1] = o2[1];
              }
            }
          };
          uint32_t v[32];
          dequant(0, v);
          wait_probed(free_, s_free_at + p.s * 8, p.ph, &s_fail, a.err);
          tc_fence_after();
          tmem_st_x32(at, v);
          const uint32_t empty = s_wempty_at + r.s * 8;
          r.next(2, SP);
          const bool more = i + kGroups < n;
          const uint32_t full_ = more ? mbar_probe_addr(s_wfull_at + r.s * 8, r.ph) : 1u;
          dequant(1, v);
          tmem_st_x32(at + 32, v);
          __syncwarp();
          if (lane == 0) arrive(empty);                  // all words have been used: their place may be filled again
          // The next words are fetched under the stores' way to tensor memory if they are here.  If not, they are waited for when they are
          // used: their place may hold a unit of the next tile, which is not used before all of this tile's have been multiplied.
          loaded = more && __all_sync(0xffffffffu, full_);
          if (loaded) load();
          tc_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) arrive(s_stored_at + p.s * 8);
          p.next(kGroups, kPlaces);
        }
        // ---- the block's part of a tile
        const int b0 = a.cut.block_of(ct * U), b1 = a.cut.block_of(ct * U + U - 1);
        // a block has at most two parts that others read: of its first tile and of its last
        auto part_of = [&](int tile, int b) {
          return a.o.partials + static_cast<size_t>(2 * b + (a.cut.start(b) < tile * U ? 1 : 0)) * M * kTileN;
        };
        auto finish = [&](int tile, int c0, int c1, int own) {
          finish_tile<EPI>(a.o, tile, warp, lane, c0, c1, own, sums, [&](int b) { return part_of(tile, b); });
        };
        float* const mine = part_of(ct, blockIdx.x) + ch;
        constexpr int T = NT / kGroups;                  // tokens of this warp
        const bool both = end - begin > 1;
        const int h0 = begin & 1, m0 = grp * T;
#pragma unroll
        for (int h = 0; h < 2; ++h)
          if (both || h == h0) {
            wait_warp(smem_u32(&s_done[h]), used[h] & 1, &s_fail, a.err);
            ++used[h];
          }
        tc_fence_after();
        float acc[T];
        {
          uint32_t v[T], w[T] = {};
          tmem_ld<T>(tmem + (both ? 0 : h0) * C::kDCols + lanes + m0, v);
          if (both) tmem_ld<T>(tmem + C::kDCols + lanes + m0, w);      // (else the other issuer may be in the next tile)
          tc_wait_ld();
#pragma unroll
          for (int j = 0; j < T; ++j) acc[j] = __uint_as_float(v[j]) + __uint_as_float(w[j]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (both || h0 == 0) arrive(smem_u32(&s_drained[0]));
          if (both || h0 == 1) arrive(smem_u32(&s_drained[1]));
        }
        __syncwarp();
        if (a.cluster) {
          // ---- the blocks of a cluster finalise some rows each, and send each other theirs
#pragma unroll
          for (int j = 0; j < T; ++j) sums[(m0 + j) * kTileN + ch] = acc[j];
          fence_proxy_async();
          named_bar_sync(2, kDqThreads);
          cluster_wait();
          const int rank = blockIdx.x - b0, first = rank * a.rows, rows = min(a.rows, M - first);
          if (warp == 0 && lane < a.cluster) {
            const int theirs = min(a.rows, M - lane * a.rows);
            if (lane == rank)
              mbar_arrive_expect_tx(s_taken, rows > 0 ? (a.cluster - 1) * rows * (kTileN * 4) : 0);
            else if (theirs > 0)
              send_cluster(mapa_shared(smem_u32(sums) + C::kSumBytes + (rank < lane ? rank : rank - 1) * theirs * (kTileN * 4), lane),
                           smem_u32(sums + lane * a.rows * kTileN), theirs * (kTileN * 4), mapa_shared(smem_u32(s_taken), lane));
          }
          __syncwarp();
          pdl_wait();
          wait_warp(smem_u32(s_taken), 0, &s_fail, a.err);
          cluster_arrive_relaxed();                      // what was sent to this block is here
          // (short loops: what runs once runs as fast as its instructions are fetched)
          constexpr int kRows = kSilu ? 2 : 1;
          const int c = kSilu ? (lane & 15) * 4 : lane * 4;
          const int n1 = EPI == kEpiRopeKv ? rope_partner(a.o.fe, ct * kTileN + c) : 0;
          const int pc = kSilu ? c + kTileN / 2 : n1 <= 0 ? 0 : n1 - ct * kTileN;
#pragma unroll 1
          for (int r = warp * kRows; r < rows; r += kDqWarps * kRows) {
            const int mine_r = kSilu ? min(r + (lane >> 4), rows - 1) : r;
            const float *near = sums + (first + mine_r) * kTileN, *far = sums + C::kSumBytes / 4 + mine_r * kTileN;
            float a0[4] = {0.f, 0.f, 0.f, 0.f}, a1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
            for (int b = 0; b < a.cluster; ++b) {
              const float* row = b == rank ? near : far;
              add4(a0, *reinterpret_cast<const float4*>(row + c));
              if (kPairs) add4(a1, *reinterpret_cast<const float4*>(row + pc));
              if (b != rank) far += rows * kTileN;
            }
            finish_row<EPI>(a.o, ct, lane, first + r, first + rows, a0, a1);
          }
          cluster_wait();
          break;
        }
        if (!waited) pdl_wait();
        waited = true;
        const bool shared = b0 != b1, last = ct == last_tile;
        if (shared && last && a.cut.whole) asm volatile("bar.sync 3, %0;" ::"n"(kDqThreads + 32) : "memory");
        if (!shared || (last && s_alone)) {
#pragma unroll
          for (int j = 0; j < T; ++j) sums[(m0 + j) * kTileN + ch] = acc[j];
          named_bar_sync(2, kDqThreads);
          finish(ct, b0, b1, blockIdx.x);
          if (!last) named_bar_sync(2, kDqThreads);      // the sums have been read
        } else {
#pragma unroll
          for (int j = 0; j < T; ++j)
            if (m0 + j < M) mine[(m0 + j) * kTileN] = acc[j];
          __syncwarp();
          if (lane == 0) arrive(smem_u32(s_written));
          __syncwarp();
        }
        if (last && (share_first || share_last)) {
          if (!shared && a.cut.whole) asm volatile("bar.sync 3, %0;" ::"n"(kDqThreads + 32) : "memory");
          asm volatile("bar.sync 4, %0;" ::"n"(kDqThreads + 32) : "memory");
          if (s_last) finish(ct, b0, b1, kNone);
          if (s_first_last) finish(first_tile, a.cut.block_of(first_tile * U), a.cut.block_of(first_tile * U + U - 1), kNone);
        }
      }
    }
  }
  __syncwarp();
  if (a.cluster && warp >= kDqWarps) {
    cluster_wait();
    cluster_arrive_relaxed();
    cluster_wait();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(s_tmem, 512);
  }
}

// Clusters of `size` blocks of this kernel that fit at once (the same on every B200).  What can't be found out is 0, and asked again.
template <int BITS, int NT, int EPI>
static int clusters_at_once(int size) {
  static std::atomic<int> known[9];
  int v = known[size].load(std::memory_order_relaxed);
  if (!v) {
    v = max_active_clusters(wna16_ts_kernel<BITS, NT, EPI>, dim3(size * (sm_count() / size)), dim3(kThreads), Cfg<BITS, NT>::kAlloc,
                            dim3(size, 1, 1));
    known[size].store(v, std::memory_order_relaxed);
  }
  return v;
}

// Ranges cut anywhere, for what takes no clusters.
static int cut_of(const WnaParams& p, UnitCut& cut) {
  int most = sm_count();
  if (most > kSkSlotCols / (2 * kTileN)) most = kSkSlotCols / (2 * kTileN);        // two parts per block
  return cut_parts(p.N / kTileN, p.K / kUnitK, 0, most, cut);
}
// The number of blocks; cluster: how many of them share a tile and meet in shared memory (0: ranges cut anywhere, or a tile each).
template <int BITS, int NT, int EPI>
static int plan(const WnaParams& p, UnitCut& cut, int& cluster) {
  const int tiles = p.N / kTileN, U = p.K / kUnitK;
  cluster = 0;
  int grid = cut_of(p, cut);
  if (EPI == kEpiPushPeers || grid <= 0) return grid;
  // As many parts as there are clusters for (B200: 74 of 2, 45 of 3, 33 of 4, 26 of 5, 22 of 6, 15 of 7 or 8).  Ranges cut anywhere leave no
  // SM idle, but a meeting through the L2 costs as much as kMeet units more than one in a cluster.
  constexpr int kMeet = BITS == 4 ? 9 : 6;
  int parts = U < 8 ? U : 8;
  while (parts > 1 && clusters_at_once<BITS, NT, EPI>(parts) < tiles) --parts;
  if (tiles * parts > sm_count() || (U + parts - 1) / parts > cut.share + (cut.rest ? 1 : 0) + kMeet) return grid;
  cluster = parts > 1 ? parts : 0;
  return cut_parts(tiles, U, parts, 0, cut);
}

// Whether the tile-split kernel (wna16_tc_dec.cu) is the faster one for a call that would be cut so here.  It is a matter of the units that a
// block takes there and here: there all blocks run at once or not, a block stores its results itself where a tile is one block's and the
// epilogue is plain, and parts meet in memory; here parts meet in clusters, or in memory for `gain` units more.  1298 plain products, 1092 with
// SiLU and 776 with a residual, K 128 - 28672, N 1024 - 65536, 1 - 64 tokens: by this rule 20 take more than 1.025 times the faster of the two
// (1.09 at most); by this kernel alone 484, 20 and 39 of them (128 x 1024, 9 tokens, here and there 2.4 / 1.9 us; 14336 x 1024, 8-bit, 32
// tokens 16.4 / 8.6; 4096 x 12800, 32 tokens 14.4 / 13.0; 4096 x 9728 11.9 / 12.1); by the other one 689, 1039 and 723.
template <int BITS, int NT, int EPI>
static bool tile_split_is_faster(const WnaParams& p, const UnitCut& cut, int cluster) {
  const int tiles = p.N / kTileN, U = p.K / kUnitK;
  // (these would go to wna16_mma.cu and wna16_sk.cu)
  if (p.M <= 16 && static_cast<int64_t>(tiles) * U >= (BITS == 4 ? 4096 : 32 * sm_count())) return false;
  const int chunks = wna16_tc_dec_turn(p);
  if (!chunks) return false;
  const bool unsplit = chunks * kChunkK >= p.K, direct = unsplit && EPI == B200_EPI_NONE;
  const int mine = cut.share + (cut.rest ? 1 : 0);
  const int less = chunks - 2 * mine;                      // half units that a block takes less here than there
  if (cluster) return direct && mine == 1 && NT <= 32;
  if (!cut.whole) return direct && (BITS == 8 || (U <= 12 && NT <= 32));      // a tile each, as there
  if (tiles * 10 < cut.parts) return true;                 // sums of more than ten parts
  if (EPI == B200_EPI_SILU_MUL) return BITS == 8 && NT == 16 && less < 2 * 11;
  if (unsplit && !direct) return false;
  const int gain = direct ? (BITS == 4 ? (NT <= 32 ? 13 : 18) : NT == 16 ? 17 : 22) : BITS == 8 && NT == 32 ? 14 : 10;
  return less < 2 * gain;
}

template <int BITS, int NT, int EPI>
static bool launch_epi(const WnaParams& p, cudaStream_t st, bool force) {
  using C = Cfg<BITS, NT>;
  Args a;
  static OncePerDevice sized;
  int device = -1;
  cudaGetDevice(&device);
  const cudaError_t e = sized(device, [] {
    return cudaFuncSetAttribute(wna16_ts_kernel<BITS, NT, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kAlloc);
  });
  if (e != cudaSuccess) {
    set_error(2, cudaGetErrorString(e));
    return true;
  }
  a.bp = reinterpret_cast<const uint8_t*>(p.bp);
  a.scales = p.scales; a.qzeros = p.qzeros;
  a.err = wait_error_flag();
  if (!a.err) return false;
  a.M = p.M; a.K = p.K; a.N = p.N; a.qfmt = p.qfmt;
  a.gshift = 30;
  if (p.group_size < p.K)
    for (int s = 0; s < 24; ++s)
      if ((kUnitK << s) == p.group_size) a.gshift = s;
  a.U = p.K / kUnitK;
  const int grid = plan<BITS, NT, EPI>(p, a.cut, a.cluster);
  if (!force && tile_split_is_faster<BITS, NT, EPI>(p, a.cut, a.cluster)) return false;
  a.by_U = unit_div(a.U);
  a.rows = a.cluster ? (p.M + a.cluster - 1) / a.cluster : p.M;
  a.o.counters = reinterpret_cast<uint32_t*>(p.workspace);
  a.o.partials = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(p.workspace) + kCounterBytes);
  a.o.bias = p.bias; a.o.c = p.c;
  a.o.M = p.M; a.o.N = p.N; a.o.splits = 0; a.o.epilogue = p.epilogue;
  if (p.fe) a.o.fe = *p.fe; else memset(&a.o.fe, 0, sizeof(a.o.fe));
  CUtensorMap xmap, wmap;
  const uint32_t es[4] = {1, 1, 1, 1};
  {
    const uint64_t dims[3] = {64, static_cast<uint64_t>(p.M), static_cast<uint64_t>(p.K / 64)};
    const uint64_t strides[2] = {static_cast<uint64_t>(p.K) * 2, 128};
    const uint32_t box[3] = {64, NT, 2};
    if (encode_tensor_map(&xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<__half*>(p.a), dims, strides, box, es,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B) != CUDA_SUCCESS) {
      set_error(2, "wna16_ts: cuTensorMapEncodeTiled failed");
      return true;
    }
  }
  wmap = xmap;
  if (EPI == B200_EPI_SILU_MUL) {
    const uint64_t subs = static_cast<uint64_t>(p.K) * BITS / 128;                   // rows of 16 bytes per channel
    const uint64_t dims[4] = {256, 2, subs, static_cast<uint64_t>(p.N / kTileN)};
    const uint64_t strides[3] = {1024, 2048, subs * 2048};
    const uint32_t box[4] = {256, 1, kUnitK * BITS / 128, 1};
    if (encode_tensor_map(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, const_cast<uint32_t*>(p.bp), dims, strides, box, es,
                          CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B) != CUDA_SUCCESS) {
      set_error(2, "wna16_ts: cuTensorMapEncodeTiled (weights) failed");
      return true;
    }
  }
  launch_pdl_cluster(wna16_ts_kernel<BITS, NT, EPI>, dim3(grid), dim3(kThreads), C::kAlloc, st, dim3(a.cluster ? a.cluster : 1), xmap, wmap, a);
  B200_CUDA_LAUNCH_CHECK();
  return true;
}

template <int BITS, int NT>
static bool launch_nt(const WnaParams& p, cudaStream_t st, bool force) {
  switch (p.epilogue) {
    case B200_EPI_SILU_MUL: return launch_epi<BITS, NT, B200_EPI_SILU_MUL>(p, st, force);
    case kEpiResidNorm: return launch_epi<BITS, NT, kEpiResidNorm>(p, st, force);
    case kEpiRopeKv: return launch_epi<BITS, NT, kEpiRopeKv>(p, st, force);
    case kEpiPushPeers: return launch_epi<BITS, NT, kEpiPushPeers>(p, st, force);
    default: return launch_epi<BITS, NT, B200_EPI_NONE>(p, st, force);
  }
}

}  // namespace ts

// Decode batches: false when the call needs another kernel.  `force`: whether or not it is the faster one.
// Up to 8 tokens 4-bit weights stay with wna16_mma.cu, which sums in another order (one token, here and there: 4096 x 28672 18.2 / 20.4 us,
// 14336 x 4096 11.5 / 12.1, 4096 x 4096 5.9 / 5.9).  From 9 on this kernel is faster at 16 / 32 / 64 tokens (here and the faster of the others:
// 4096 x 28672 18.4 / 25.5, 19.5 / 30.2, 23.1 / 36.7; 14336 x 4096 11.7 / 13.3, 12.0 / 13.6, 12.8 / 16.7; 2048 x 2048 4.2 / 5.6, 4.5 / 5.9,
// 5.2 / 9.5), but for many short tiles, where a block finalises two or three (16 tokens: 2048 x 34816 14.8 / 14.4, 512 x 131072 19.9 / 17.0,
// though 1024 x 65536 15.8 / 16.5; 8-bit, 32 tokens, 2048 x 34816 18.4 / 17.0): those stay where they were, at up to 16 tokens with
// wna16_mma.cu and wna16_sk.cu, which take no others of these by themselves.  8-bit weights, 1 / 16 / 32 tokens: 4096 x 28672 24.1 / 26.9,
// 25.1 / 28.6, 26.6 / 30.7, 14336 x 4096 14.0 / 15.0, 14.4 / 15.5, 15.0 / 16.7, 4096 x 4096 6.7 / 7.5, 7.0 / 8.0, 7.4 / 8.7; with 64 tokens
// the rings would be too short (14336 x 4096 19.4 / 17.3).  tile_split_is_faster has the sizes at which it is the tile-split kernel's turn.
bool launch_wna16_ts(const WnaParams& p, cudaStream_t st, bool force) {
  if (p.M > (p.bits == 4 ? 64 : 32) || p.K % ts::kUnitK != 0 || p.N % kTileN != 0 || p.no_split) return false;
  const int64_t tiles = p.N / kTileN, U = p.K / ts::kUnitK;
  if (!force && ((p.bits == 4 && p.M <= 8) || (U <= 16 && tiles * U >= 4096) || (p.M <= 32 && wna16_sk_first()))) return false;
  if (p.group_size < p.K) {                  // a unit lies in one group, whose index is a shift of the unit's
    bool ok = false;
    for (int s = 0; s < 24; ++s) ok = ok || (ts::kUnitK << s) == p.group_size;
    if (!ok) return false;
  }
  // 16-byte copies (scales and zero points are read one by one, but calls with such views keep their kernels); four results and
  // bias values at a time
  const uintptr_t low = reinterpret_cast<uintptr_t>(p.bp) | reinterpret_cast<uintptr_t>(p.scales) |
                        reinterpret_cast<uintptr_t>(p.qzeros) | reinterpret_cast<uintptr_t>(p.a) |
                        reinterpret_cast<uintptr_t>(p.workspace);
  if (low & 15) return false;
  if ((reinterpret_cast<uintptr_t>(p.bias) | reinterpret_cast<uintptr_t>(p.c)) & 7) return false;
  if (p.epilogue == B200_EPI_SILU_MUL && (tiles & 1)) return false;
  if (p.epilogue == kEpiRopeKv && p.fe && (kTileN % p.fe->D) != 0) return false;
  if (U * p.N >= int64_t{1} << 31) return false;             // offsets of scales
  UnitCut cut;
  if (ts::cut_of(p, cut) <= 0) return false;
  if (p.bits == 4) return p.M <= 16 ? ts::launch_nt<4, 16>(p, st, force) : p.M <= 32 ? ts::launch_nt<4, 32>(p, st, force) : ts::launch_nt<4, 64>(p, st, force);
  return p.M <= 16 ? ts::launch_nt<8, 16>(p, st, force) : ts::launch_nt<8, 32>(p, st, force);
}

}  // namespace b200
