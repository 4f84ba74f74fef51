// W4A16 GEMM of decode batches: every warp streams, dequantises and multiplies its own weights.
//
// The reference's arithmetic: weights (q - z) * s rounded once to fp16, fp32 sums.
//
// What bounds it.  The weights' HBM time is 22 SM cycles per scheduler and 256 weights (at 6.5 TB/s and 1.9 GHz); one
// mma.sync.m16n8k16 takes a scheduler's tensor pipe 8 cycles and multiplies 256 weights with 8 tokens; the thirteen
// instructions that turn 256 packed weights into an A fragment take 16 cycles of the fp16 pipe.  They overlap in part only,
// so up to 16 tokens the memory can be kept fairly busy, provided that nothing else costs issue slots: no tensor memory, no
// hand-over of dequantised weights, one wait per 128 weights of K.  The rest is fixed time per launch: the activations'
// way to shared memory, the meeting of a tile's parts, code fetched cold (loops that run once per tile are not unrolled).
//
// Layout.  A weight tile of the tile-major format holds 32 consecutive K of a channel in 16 bytes, so the
// four lanes that share a row of an A fragment take 16 bytes each: together 128 K, one quantisation group or part of one.
// Which K a fragment column stands for does not matter as long as both operands agree.  A warp has two blocks of 16
// channels (fragment rows g <-> channel 2g, g + 8 <-> channel 2g + 1), chosen so that gate and up, or the two halves of a
// rotated head, meet in the same lane: every epilogue works on registers.
//
// Work.  A unit is a tile of 128 channels x 128 K.  Eight warps per block = two groups of four, each with every second
// unit of the block's range; ranges are cut evenly over the grid (a tile may be cut anywhere between units).  A unit's
// weights, scales, zero points (bulk copies) and activations (TMA) arrive in a ring of the group; weights never wait for
// the previous kernel.  Registers and shared memory leave room for two blocks per SM.
#include <cstring>

#include "host/per_device.hpp"
#include "host/unit_cut.hpp"
#include "wna16.cuh"

namespace b200 {
namespace wm {

constexpr int kUnitK = 128;
constexpr int kThreads = 256;
constexpr int kKG = 2;                       // K groups of a block
constexpr int kGW = 4;                       // warps of a group: 32 channels each
constexpr int kGThreads = kGW * 32;
static_assert(kKG * kGThreads == kThreads && kGW * 32 == kTileN, "block shape");

// Where sub-row t of a chunk starts: the shift keeps the four lanes of a fragment's row (and two rows) on different banks.
__host__ __device__ constexpr int sub_off(int t) { return t * (kTileN * 16) + ((t & 1) ? 16 : 0) + ((t & 2) ? 64 : 0); }

template <int NT>
struct Cfg {
  static constexpr int kWeightBytes = sub_off(3) + kTileN * 16 + 48; // of a unit, a multiple of 128
  static constexpr int kBox = NT * 8 * 128;                          // 64 K of the activations, 128-byte swizzle
  static constexpr int kXOff = 0;                                    // two boxes, the second shifted by two rows
  static constexpr int kWOff = 2 * kBox + 256;
  static constexpr int kSOff = kWOff + kWeightBytes;
  static constexpr int kScaleBytes = kTileN * 2, kZeroBytes = kTileN / 2;
  static constexpr int kZOff = kSOff + kScaleBytes;
  static constexpr int kStage = (kZOff + kZeroBytes + 1023) / 1024 * 1024;
  static constexpr uint32_t kTx = 4 * kTileN * 16 + 2 * kBox + kScaleBytes;      // + kZeroBytes
  static constexpr int kHand = kGW * NT * 512;                       // half of the sums that the second group hands over
  // two blocks per SM where three units per group fit into half of the shared memory
  static constexpr int kHalf = 113 * 1024 - 2048;
  static constexpr int kFit = (kHalf - kHand) / (kKG * kStage);
  static constexpr int kStages = kFit >= 5 ? 5 : kFit >= 3 ? kFit : 3;
  static constexpr int kLag = kStages > 3 ? 2 : 1;                   // a unit's place is filled again so many units later
  static constexpr int kHandOff = kKG * kStages * kStage;
  static constexpr int kAlloc = kHandOff + kHand + 1024;             // the start is aligned to 1024 bytes
  static constexpr int kBlocks = kAlloc <= kHalf + 1024 ? 2 : 1;     // per SM
  static_assert(kAlloc <= 220 * 1024, "shared memory");
};

struct Args {
  const uint8_t* bp;
  const __half* scales;
  const uint32_t* qzeros;
  float* partials;
  uint32_t* counters;
  int* err;              // set by a wait that gave up
  int M, K, N, qfmt;
  int gshift;            // log2(group_size / 128); 30: one group
  int U;                 // units per tile
  UnitCut cut;
  UnitDiv by_U;
  int hd_shift;          // log2(head_dim / 2) of the rotated epilogue
  SplitOut o;
};

__device__ __forceinline__ void mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                    uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// 4-bit word -> fp16((q - z) * s) of k (0,1) (2,3), or (4,5) (6,7).  zlo = half2(1024 + z), zhi = -half2(64 + z)
__device__ __forceinline__ void dq4_half(uint32_t x, int half, uint32_t zlo, uint32_t zhi, __half2 s, uint32_t (&v)[2]) {
  const uint32_t y = half ? x >> 8 : x;
  const __half2 lo = __hsub2(u32_as_h2(lop3_or_and(y, 0x000F000Fu, 0x64006400u)), u32_as_h2(zlo));
  const __half2 hi = __hfma2(u32_as_h2(lop3_or_and(y, 0x00F000F0u, 0x64006400u)), __float2half2_rn(0.0625f), u32_as_h2(zhi));
  v[0] = h2_as_u32(__hmul2(lo, s));
  v[1] = h2_as_u32(__hmul2(hi, s));
}
// First channels of the two blocks of 16 that warp w of a group has in a tile.
template <int EPI>
__device__ __forceinline__ void channels(int tile, int w, int N, int hd_shift, int& ca, int& cb) {
  if (EPI == B200_EPI_SILU_MUL) {                        // a tile = 64 gate channels and their 64 up channels
    ca = tile * (kTileN / 2) + w * 16;
    cb = ca + (N >> 1);
  } else if (EPI == kEpiRopeKv) {                        // d and d + D / 2 of a head
    const int hd = 1 << hd_shift;
    ca = tile * kTileN + ((w * 16 >> hd_shift) << (hd_shift + 1)) + (w * 16 & (hd - 1));
    cb = ca + hd;
  } else {
    ca = tile * kTileN + w * 32;
    cb = ca + 16;
  }
}

__device__ __forceinline__ float2 half2_at(const __half* p) {
  return __half22float2(*reinterpret_cast<const __half2*>(p));
}
__device__ __forceinline__ void put_half2(__half* p, float a, float b) {
  *reinterpret_cast<__half2*>(p) = __floats2half2_rn(a, b);
}
__device__ __forceinline__ float round16(float v) { return __half2float(__float2half_rn(v)); }

// Finalises a tile: tot[block][token tile][0, 1 | 2, 3] = channel 2g | 2g + 1 of the block, tokens 2t, 2t + 1.  Called by
// the four warps of a group; rs: the rows' factors (shared memory), sq: [4][NT * 8] floats of shared memory.
template <int EPI, int NT>
__device__ __forceinline__ void finish_tile(const SplitOut& o, int tile, int w, int lane, const float (&tot)[2][NT][4],
                                            const float* rs, float* sq, int bar_id, int hd_shift) {
  const FusedEpi& fe = o.fe;
  const int g = lane >> 2, t = lane & 3, M = o.M, N = o.N;
  int ca, cb;
  channels<EPI>(tile, w, N, hd_shift, ca, cb);
  ca += 2 * g;
  cb += 2 * g;
  float2 ba = make_float2(0.f, 0.f), bb = ba, na = ba, nb = ba;
  if (o.bias) {
    ba = half2_at(o.bias + ca);
    bb = half2_at(o.bias + cb);
  }
  if (EPI == kEpiResidNorm) {
    na = half2_at(fe.norm_w + ca);
    nb = half2_at(fe.norm_w + cb);
  }
  // one copy of the code below for all token tiles: it runs once per tile and is fetched cold, so its length is its time
  float fin[NT * 2][4];
#pragma unroll
  for (int i = 0; i < NT * 2; ++i) {
    fin[i][0] = tot[0][i >> 1][i & 1];
    fin[i][1] = tot[0][i >> 1][2 + (i & 1)];
    fin[i][2] = tot[1][i >> 1][i & 1];
    fin[i][3] = tot[1][i >> 1][2 + (i & 1)];
  }
#pragma unroll 1
  for (int i = 0; i < NT * 2; ++i) {
    const int m = (i >> 1) * 8 + 2 * t + (i & 1);
    const bool valid = m < M;
    const float f = fe.ssq_in && valid ? rs[m] : 1.f;
    const float a0 = fin[i][0] * f + ba.x, a1 = fin[i][1] * f + ba.y;
    const float b0 = fin[i][2] * f + bb.x, b1 = fin[i][3] * f + bb.y;
    if (EPI == B200_EPI_SILU_MUL) {
      if (valid) {
        // round the two GEMM outputs to fp16 first: the values an unfused pipeline would see
        const float g0 = round16(a0), g1 = round16(a1);
        put_half2(o.c + static_cast<size_t>(m) * (N >> 1) + ca, g0 / (1.f + __expf(-g0)) * round16(b0),
                  g1 / (1.f + __expf(-g1)) * round16(b1));
      }
    } else if (EPI == kEpiResidNorm) {
      float s = 0.f;
      if (valid) {
        // llama.rs:126-130: the GEMM output is fp16, the residual add is done in fp16
        const size_t row = static_cast<size_t>(m) * N;
        const float2 ra = half2_at(fe.resid + row + ca), rb = half2_at(fe.resid + row + cb);
        const float x0 = round16(ra.x + round16(a0)), x1 = round16(ra.y + round16(a1));
        const float x2 = round16(rb.x + round16(b0)), x3 = round16(rb.y + round16(b1));
        put_half2(fe.resid + row + ca, x0, x1);
        put_half2(fe.resid + row + cb, x2, x3);
        put_half2(o.c + row + ca, x0 * na.x, x1 * na.y);
        put_half2(o.c + row + cb, x2 * nb.x, x3 * nb.y);
        s = x0 * x0 + x1 * x1 + x2 * x2 + x3 * x3;
      }
      s += __shfl_xor_sync(0xffffffffu, s, 4);
      s += __shfl_xor_sync(0xffffffffu, s, 8);
      s += __shfl_xor_sync(0xffffffffu, s, 16);
      if (g == 0) sq[w * (NT * 8) + m] = s;
    } else if (EPI == kEpiRopeKv) {
      if (valid) {
        const int D = fe.D, hh = ca >> (hd_shift + 1), d = ca & (D - 1);     // one head for both blocks, d < D / 2
        const bool is_v = hh >= fe.H + fe.Hkv;
        float oa0 = a0, oa1 = a1, ob0 = b0, ob1 = b1;
        if (!is_v) {
          // the reference rotates the fp16 GEMM outputs (rotary_emb.rs:88-104)
          const size_t ci = (static_cast<size_t>(fe.positions[m]) << hd_shift) + d;
          const float2 cs = half2_at(fe.cos + ci), sn = half2_at(fe.sin + ci);
          const float x0 = round16(a0), x1 = round16(a1), y0 = round16(b0), y1 = round16(b1);
          oa0 = x0 * cs.x - y0 * sn.x;
          oa1 = x1 * cs.y - y1 * sn.y;
          ob0 = y0 * cs.x + x0 * sn.x;
          ob1 = y1 * cs.y + x1 * sn.y;
        }
        if (hh < fe.H) {
          put_half2(o.c + static_cast<size_t>(m) * N + ca, oa0, oa1);       // q stays in the fused buffer
          put_half2(o.c + static_cast<size_t>(m) * N + cb, ob0, ob1);
        } else {
          const int sl = static_cast<int>(fe.slots[m]);
          if (sl >= 0) {
            __half* cache = is_v ? fe.v_cache : fe.k_cache;
            const int kvh = hh - fe.H - (is_v ? fe.Hkv : 0);
            const size_t ci = (static_cast<size_t>(sl) * fe.Hkv + kvh) * D + d;
            if (fe.kv_fp8) {
              __half2_raw p = __floats2half2_rn(oa0, oa1), q = __floats2half2_rn(ob0, ob1);
              uint8_t* c8 = reinterpret_cast<uint8_t*>(cache) + ci;
              *reinterpret_cast<uint16_t*>(c8) = __nv_cvt_halfraw2_to_fp8x2(p, __NV_SATFINITE, __NV_E4M3);
              *reinterpret_cast<uint16_t*>(c8 + (D >> 1)) = __nv_cvt_halfraw2_to_fp8x2(q, __NV_SATFINITE, __NV_E4M3);
            } else {
              put_half2(cache + ci, oa0, oa1);
              put_half2(cache + ci + (D >> 1), ob0, ob1);
            }
          }
        }
      }
    } else if (EPI == kEpiPushPeers) {
      if (valid) {
        const size_t row = static_cast<size_t>(m) * N;
#pragma unroll 1
        for (int p = 0; p < fe.push_world; ++p) {                           // peer-mapped (NVLink) stores
          put_half2(fe.push[p] + row + ca, a0, a1);
          put_half2(fe.push[p] + row + cb, b0, b1);
        }
      }
    } else if (valid) {
      put_half2(o.c + static_cast<size_t>(m) * N + ca, a0, a1);
      put_half2(o.c + static_cast<size_t>(m) * N + cb, b0, b1);
    }
  }
  if (EPI == kEpiResidNorm) {
    named_bar_sync(bar_id, kGThreads);
    const int m = w * 32 + lane;
    if (m < M) {
      constexpr int S = NT * 8;
      fe.ssq_out[m * kSsqStride + tile] = (sq[m] + sq[S + m]) + (sq[2 * S + m] + sq[3 * S + m]);
    }
    named_bar_sync(bar_id, kGThreads);       // sq is free for the next tile
  }
  if (EPI == kEpiPushPeers) push_signal(fe, w * 32 + lane, kGThreads, bar_id);
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

template <int NT, int EPI>
__global__ void __launch_bounds__(kThreads, Cfg<NT>::kBlocks)
wna16_mma_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ Args a) {
  using C = Cfg<NT>;
  constexpr int S = C::kStages;
  constexpr bool kSilu = EPI == B200_EPI_SILU_MUL;
  extern __shared__ uint8_t smem_raw[];
  __shared__ float s_rs[NT * 8], s_sq[4 * NT * 8];
  __shared__ uint64_t s_full[kKG * S], s_empty[kKG * S];
  __shared__ int s_flag, s_fail;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int kg = warp >> 2, w = warp & 3, g = lane >> 2, t = lane & 3;
  const int gt = threadIdx.x & (kGThreads - 1);
  const int bar_id = 1 + kg;                 // barriers 1, 2: the groups; 3, 4: the hand-over's place is full, empty
  const int U = a.U, N = a.N, M = a.M, K = a.K;
  const int u0 = a.cut.start(blockIdx.x), u1 = a.cut.start(blockIdx.x + 1);
  const int first_tile = a.by_U(u0), last_tile = a.by_U(u1 - 1);
  uint8_t* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  uint8_t* ring = smem + kg * (S * C::kStage);
  const uint32_t ring_at = smem_u32(ring);
  const uint32_t full = smem_u32(s_full + kg * S), empty = smem_u32(s_empty + kg * S);
  pdl_trigger();
  if (threadIdx.x == 0) {
    for (int i = 0; i < kKG * S; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&s_empty[i], kGW);
    }
    s_fail = 0;
    fence_barrier_init();
    prefetch_tmap(&xmap);
  }

  // ---- copies.  The lanes of one warp bring a unit: lanes 0 .. its sub-rows (with SiLU half of them gate, half up), then the
  // scales, then the zero points; lanes 30 and 31 the activations.
  constexpr int kRuns = kSilu ? 2 : 1;
  constexpr int kSubs = 4;                    // of 32 K each
  const uint8_t* c_src = nullptr;            // of tile 0, unit 0
  uint32_t c_dst = 0, c_bytes = 0;
  size_t c_tile = 0;                         // bytes from tile to tile, from unit to unit (from group to group)
  uint32_t c_odd = 0, c_unit = 0;
  int c_shift = 0, c_half = 0;
  {
    const size_t tile_bytes = static_cast<size_t>(K) * kTileN / 2;
    const int zb = C::kZeroBytes / kRuns, sb = C::kScaleBytes / kRuns;
    if (lane < kSubs * kRuns) {
      const int sub = lane % kSubs, run = lane / kSubs;
      c_src = a.bp + run * (N / kTileN / 2) * tile_bytes + sub * (kTileN * 16);
      c_bytes = kTileN * 16 / kRuns;
      c_dst = C::kWOff + sub_off(sub) + run * (kTileN * 8);
      c_tile = tile_bytes;
      c_unit = kUnitK * kTileN / 2;
      if (kSilu) {                           // two tiles of 64 + 64 channels share a weight tile
        c_half = 1;
        c_odd = kTileN * 8;
      }
    } else if (lane < kSubs * kRuns + kRuns) {
      const int run = lane - kSubs * kRuns;
      c_src = reinterpret_cast<const uint8_t*>(a.scales) + static_cast<size_t>(run) * N;
      c_bytes = sb;
      c_dst = C::kSOff + run * sb;
      c_tile = sb;
      c_unit = N * 2;
      c_shift = a.gshift;
    } else if (lane < kSubs * kRuns + 2 * kRuns && a.qzeros) {
      const int run = lane - kSubs * kRuns - kRuns;
      c_src = reinterpret_cast<const uint8_t*>(a.qzeros) + static_cast<size_t>(run) * N / 4;
      c_bytes = zb;
      c_dst = C::kZOff + run * zb;
      c_tile = zb;
      c_unit = N / 2;
      c_shift = a.gshift;
    }
  }
  const uint32_t tx = C::kTx + (a.qzeros ? C::kZeroBytes : 0);
  auto copy_weights = [&](int st, int tile, int u) {
    const uint32_t bar = full + st * 8;
    if (lane == 0) asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(tx) : "memory");
    __syncwarp();
    if (c_bytes)
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       ring_at + st * C::kStage + c_dst),
                   "l"(c_src + static_cast<size_t>(tile >> c_half) * c_tile + (tile & 1) * c_odd +
                       static_cast<size_t>(u >> c_shift) * c_unit),
                   "r"(c_bytes), "r"(bar)
                   : "memory");
  };
  auto copy_x = [&](int st, int u) {
    if (lane >= 30) {
      const int box = lane - 30;
      asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
                       ring_at + st * C::kStage + C::kXOff + box * (C::kBox + 256)),
                   "l"(reinterpret_cast<uint64_t>(&xmap)), "r"(full + st * 8), "r"(u * kUnitK + box * 64), "r"(0)
                   : "memory");
    }
  };
  // group kg has the block's units kg, kg + 2, ..
  int unit = u0 + kg, tile = first_tile;     // the next one to bring, and its tile
  auto bring = [&](int st) {
    while (unit >= (tile + 1) * U) ++tile;
    copy_weights(st, tile, unit - tile * U);
  };

  __syncthreads();
  // ---- prologue: the weights of the first units before the wait for the previous kernel, their activations after it
  // (one warp per unit: issuing a copy takes far longer than an instruction)
#pragma unroll 1
  for (int s = w; s < S; s += kGW) {
    unit = u0 + kg + s * kKG;
    if (unit < u1) bring(s);
  }
  pdl_wait();
#pragma unroll 1
  for (int s = w; s < S; s += kGW) {
    const int xu = u0 + kg + s * kKG;
    if (xu < u1) copy_x(s, xu - a.by_U(xu) * U);
  }
  unit = u0 + kg + S * kKG;
  if (a.o.fe.ssq_in) {
#pragma unroll 1
    for (int m = warp; m < M; m += kThreads / 32) {
      const float v = warp_sum(ssq_lane_partial(a.o.fe.ssq_in + m * kSsqStride, a.o.fe.ssq_tiles, lane));
      if (lane == 0) s_rs[m] = rsqrtf(v * a.o.fe.inv_dim + a.o.fe.eps);
    }
  }
  __syncthreads();

  int la, lb;                                // the warp's two blocks' first channels within the tile's 128
  if (kSilu) {
    la = w * 16;
    lb = 64 + w * 16;
  } else {
    channels<EPI>(0, w, N, a.hd_shift, la, lb);
  }
  const int bd = kSilu ? 64 : EPI == kEpiRopeKv ? lb - la : 16;      // channels from one block to the other
  const uint32_t q_a = C::kWOff + sub_off(t) + (la + 2 * g) * 16, q_d = bd * 16;
  uint32_t x_at[4];
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const int box = t >> 1, piece = (t & 1) * 4 + s;
    x_at[s] = C::kXOff + box * (C::kBox + 256) + g * 128 + ((piece ^ ((g + 2 * box) & 7)) * 16);
  }
  const uint32_t sc_a = C::kSOff + (la + 2 * g) * 2, sc_d = bd * 2;
  const uint32_t z_a = C::kZOff + ((la + 2 * g) / 8) * 4, z_d = bd / 2;
  const bool awq = a.qfmt == B200_QFMT_AWQ, has_z = a.qzeros != nullptr;
  const uint32_t z_shift = awq ? 4 * (g & 3) : 8 * (g & 3);

  int st = 0, done = 0, at = u0 + kg;        // place of the unit at hand, units done, the unit
  uint32_t ph = 0;
  int refills = 0;                           // by this warp, of one place: (w - kLag) mod S
  static_assert(S == kGW, "the warps take turns as the places do");
  if (kg == 0) asm volatile("bar.arrive 4, %0;" ::"n"(kThreads) : "memory");
#pragma unroll 1
  for (int ct = first_tile; ct <= last_tile; ++ct) {
    const int t0 = ct * U, to = min(t0 + U, u1);
    float tot[2][NT][4];
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) tot[b][n][e] = 0.f;
#pragma unroll 1
    for (; at < to; at += kKG, ++done) {
      // the four warps take turns at bringing the unit that goes into the place of kLag units ago
      if (done >= C::kLag && unit < u1) {
        if ((done & 3) == w) {
          const int ds = st >= C::kLag ? st - C::kLag : st - C::kLag + S;
          if (__all_sync(0xffffffffu, wait(empty + ds * 8, st >= C::kLag ? ph : ph ^ 1, &s_fail, a.err))) {
            bring(ds);
            copy_x(ds, unit - tile * U);
            ++refills;
          }
        }
        unit += kKG;
      }
      wait(full + st * 8, ph, &s_fail, a.err);
      const uint8_t* sp = ring + st * C::kStage;
      uint32_t zlo[4], zhi[4];               // 1024 + z and -(64 + z) of the four channels
      {
        uint32_t za = 0x64086408u, zb = za;  // of two neighbouring channels, one in each half
        if (has_z) {
          const uint32_t wa = *reinterpret_cast<const uint32_t*>(sp + z_a) >> z_shift;
          const uint32_t wb = *reinterpret_cast<const uint32_t*>(sp + z_a + z_d) >> z_shift;
          if (awq) {
            za = lop3_or_and(wa, 0x000F000Fu, 0x64006400u);
            zb = lop3_or_and(wb, 0x000F000Fu, 0x64006400u);
          } else {
            za = ((wa & 0xFu) | ((wa & 0xF0u) << 12)) + 0x64016401u;
            zb = ((wb & 0xFu) | ((wb & 0xF0u) << 12)) + 0x64016401u;
          }
        }
        zlo[0] = __byte_perm(za, 0, 0x1010);
        zlo[1] = __byte_perm(za, 0, 0x3232);
        zlo[2] = __byte_perm(zb, 0, 0x1010);
        zlo[3] = __byte_perm(zb, 0, 0x3232);
#pragma unroll
        for (int r = 0; r < 4; ++r) zhi[r] = h2_as_u32(__hsub2(__float2half2_rn(960.f), u32_as_h2(zlo[r])));
      }
      auto frag = [&](uint32_t off) { return *reinterpret_cast<const uint4*>(sp + off); };
      const __half2 s_a = *reinterpret_cast<const __half2*>(sp + sc_a), s_b = *reinterpret_cast<const __half2*>(sp + sc_a + sc_d);
      const __half2 sc[4] = {__low2half2(s_a), __high2half2(s_a), __low2half2(s_b), __high2half2(s_b)};
      const uint4 w0 = frag(q_a), w1 = frag(q_a + 16), w2 = frag(q_a + q_d), w3 = frag(q_a + q_d + 16);
      const uint32_t q[4][4] = {{w0.x, w0.y, w0.z, w0.w}, {w1.x, w1.y, w1.z, w1.w}, {w2.x, w2.y, w2.z, w2.w}, {w3.x, w3.y, w3.z, w3.w}};
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        uint4 x[NT];
#pragma unroll
        for (int n = 0; n < NT; ++n) x[n] = frag(x_at[s] + n * 1024);
        if (s == 3) {
          // The last read of the unit's place.  What was read has to be there before the copies of a later unit may be asked for, and
          // these write by another proxy: without the two fences one warp in some 10^7 read the last activations after them (seen
          // at 9 - 16 tokens, 34944 x 30848: one call in 100).  They cost nothing: four projections, one token 47.1 -> 46.7 us.
          reads_done();
          __syncwarp();
          if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty + st * 8) : "memory");
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t p[4][2];
#pragma unroll
          for (int r = 0; r < 4; ++r) dq4_half(q[r][s], h, zlo[r], zhi[r], sc[r], p[r]);
#pragma unroll
          for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int b = 0; b < 2; ++b)
              mma(tot[b][n], p[2 * b][0], p[2 * b + 1][0], p[2 * b][1], p[2 * b + 1][1], h ? x[n].z : x[n].x, h ? x[n].w : x[n].y);
        }
      }
      if (++st == S) {
        st = 0;
        ph ^= 1;
      }
    }
    // ---- the block's part of a tile is done: the second group hands its sums to the first, one block of channels at a time
    float4* hand = reinterpret_cast<float4*>(smem + C::kHandOff + w * (NT * 512)) + lane;
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      if (kg == 1) {
        asm volatile("bar.sync 4, %0;" ::"n"(kThreads) : "memory");
#pragma unroll
        for (int n = 0; n < NT; ++n) hand[n * 32] = make_float4(tot[b][n][0], tot[b][n][1], tot[b][n][2], tot[b][n][3]);
        asm volatile("bar.arrive 3, %0;" ::"n"(kThreads) : "memory");
      } else {
        asm volatile("bar.sync 3, %0;" ::"n"(kThreads) : "memory");
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          const float4 v = hand[n * 32];
          tot[b][n][0] += v.x;
          tot[b][n][1] += v.y;
          tot[b][n][2] += v.z;
          tot[b][n][3] += v.w;
        }
        if (b == 0 || ct < last_tile) asm volatile("bar.arrive 4, %0;" ::"n"(kThreads) : "memory");
      }
    }
    if (kg == 1) continue;
    if (u0 > t0 || u1 < t0 + U) {
      // ---- the tile has several contributors: the last of them to arrive sums their parts in the order of K
      const int b0 = a.cut.block_of(t0), b1 = a.cut.block_of(t0 + U - 1);
      constexpr int kPart = kTileN * NT * 8;                        // floats of a part, in the lanes' own order
      // a block has at most two parts: of its first tile and of its last
      auto part_of = [&](int b) {
        return reinterpret_cast<float4*>(a.partials + static_cast<size_t>(2 * b + (a.cut.start(b) < t0 ? 1 : 0)) * kPart +
                                         w * (NT * 256)) + lane;
      };
      float4* mp = part_of(blockIdx.x);
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int n = 0; n < NT; ++n) mp[(b * NT + n) * 32] = make_float4(tot[b][n][0], tot[b][n][1], tot[b][n][2], tot[b][n][3]);
      named_bar_sync(bar_id, kGThreads);
      if (gt == 0) {
        // releases this block's part (ordered before by the barrier) and acquires the others'
        unsigned old;
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(a.counters + ct) : "memory");
        const int last = old == static_cast<unsigned>(b1 - b0) ? 1 : 0;
        if (last) a.counters[ct] = 0;                               // at rest again for the next launch
        s_flag = last;
      }
      named_bar_sync(bar_id, kGThreads);
      if (!s_flag) continue;
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) tot[b][n][e] = 0.f;
      constexpr int kBatch = 8 / NT;                                // parts on their way at a time
#pragma unroll 1
      for (int j = b0; j <= b1; j += kBatch) {
        float4 v[kBatch][2][NT];
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
          const float4* ip = part_of(min(j + i, b1));
#pragma unroll
          for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int n = 0; n < NT; ++n) v[i][b][n] = __ldcg(ip + (b * NT + n) * 32);
        }
#pragma unroll
        for (int i = 0; i < kBatch; ++i)
          if (j + i <= b1) {
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
              for (int n = 0; n < NT; ++n) {
                tot[b][n][0] += v[i][b][n].x;
                tot[b][n][1] += v[i][b][n].y;
                tot[b][n][2] += v[i][b][n].z;
                tot[b][n][3] += v[i][b][n].w;
              }
          }
      }
    }
    finish_tile<EPI, NT>(a.o, ct, w, lane, tot, s_rs, s_sq, bar_id, a.hd_shift);
  }
  // after a wait has given up: no copy may land in this memory when it is another block's
  if (*reinterpret_cast<volatile int*>(&s_fail)) {
    const int at_place = (w + S - C::kLag) % S, fills = refills + (u0 + kg + at_place * kKG < u1 ? 1 : 0);
    if (fills > 0) mbar_wait_limited(&s_full[kg * S + at_place], (fills - 1) & 1, nullptr, a.err);
  }
}

template <int NT>
static int cut_of(const WnaParams& p, UnitCut& cut) {
  int most = sm_count() * Cfg<NT>::kBlocks;
  if (most > kSkSlotCols / (2 * kTileN)) most = kSkSlotCols / (2 * kTileN);        // two parts per block
  return cut_units(p.N / kTileN, p.K / kUnitK, most, kKG, cut);
}

template <int NT, int EPI>
static bool launch_epi(const WnaParams& p, cudaStream_t st) {
  using C = Cfg<NT>;
  Args a;
  a.bp = reinterpret_cast<const uint8_t*>(p.bp);
  a.scales = p.scales; a.qzeros = p.qzeros;
  a.counters = reinterpret_cast<uint32_t*>(p.workspace);
  a.partials = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(p.workspace) + kCounterBytes);
  a.err = wait_error_flag();
  if (!a.err) return false;
  a.M = p.M; a.K = p.K; a.N = p.N; a.qfmt = p.qfmt;
  a.gshift = 30;
  if (p.group_size < p.K)
    for (int s = 0; s < 24; ++s)
      if ((kUnitK << s) == p.group_size) a.gshift = s;
  a.U = p.K / kUnitK;
  const int grid = cut_of<NT>(p, a.cut);
  a.by_U = unit_div(a.U);
  a.hd_shift = 6;
  if (p.fe && p.epilogue == kEpiRopeKv) a.hd_shift = p.fe->D == 128 ? 6 : p.fe->D == 64 ? 5 : 4;
  a.o.partials = a.partials; a.o.counters = a.counters; a.o.bias = p.bias; a.o.c = p.c;
  a.o.M = p.M; a.o.N = p.N; a.o.splits = 0; a.o.epilogue = p.epilogue;
  if (p.fe) a.o.fe = *p.fe; else memset(&a.o.fe, 0, sizeof(a.o.fe));
  CUtensorMap xmap;
  {
    const uint64_t dims[2] = {static_cast<uint64_t>(p.K), static_cast<uint64_t>(p.M)};
    const uint64_t strides[1] = {static_cast<uint64_t>(p.K) * 2};
    const uint32_t box[2] = {64, NT * 8}, es[2] = {1, 1};
    if (encode_tensor_map(&xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half*>(p.a), dims, strides, box, es,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B) != CUDA_SUCCESS) {
      set_error(2, "wna16_mma: cuTensorMapEncodeTiled failed");
      return true;
    }
  }
  static OncePerDevice sized;
  int device = -1;
  cudaGetDevice(&device);
  const cudaError_t e = sized(device, [] {
    return cudaFuncSetAttribute(wna16_mma_kernel<NT, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kAlloc);
  });
  if (e != cudaSuccess) {
    set_error(2, cudaGetErrorString(e));
    return true;
  }
  launch_pdl(wna16_mma_kernel<NT, EPI>, dim3(grid), dim3(kThreads), C::kAlloc, st, xmap, a);
  B200_CUDA_LAUNCH_CHECK();
  return true;
}

template <int NT>
static bool launch_nt(const WnaParams& p, cudaStream_t st) {
  switch (p.epilogue) {
    case B200_EPI_SILU_MUL: return launch_epi<NT, B200_EPI_SILU_MUL>(p, st);
    case kEpiResidNorm: return launch_epi<NT, kEpiResidNorm>(p, st);
    case kEpiRopeKv: return launch_epi<NT, kEpiRopeKv>(p, st);
    case kEpiPushPeers: return launch_epi<NT, kEpiPushPeers>(p, st);
    default: return launch_epi<NT, B200_EPI_NONE>(p, st);
  }
}

}  // namespace wm

// Decode batches of 4-bit weights: false when the call needs another kernel.  `force`: whether or not it is the faster one.
// Up to 8 tokens it is at every size measured.  At 9 - 16, where the products take twice the issue slots, from 4096 units on, of which
// wna16_ts.cu comes first for all but K <= 2048 (N from 32768 on) and results off 8 bytes.  us at 1 / 16 tokens, here and the faster of the other two: 4096 x 6144 7.2 / 9.3 and 8.5 / 8.9, 4096 x 4096 5.7 / 7.6 and
// 7.1 / 7.5, 4096 x 28672 21.0 / 24.9 and 25.7 / 29.1, 14336 x 4096 12.2 / 14.8 and 13.8 / 14.3, 2048 x 2560 4.5 / 6.2 and 5.4 / 6.0,
// 5632 x 2048 6.5 / 8.2 and 6.2 / 6.6, 8192 x 10240 15.6 / 18.1 and 17.9 / 20.0, 8192 x 57344 65 / 75 and 100 / 102, 28672 x 8192
// 35.8 / 41.5 and 38.3 / 41.0.  (8-bit weights stay with those: a unit is twice the bytes, one block per SM: 4096 x 28672 35 and 28.)
bool wna16_mma_takes(const WnaParams& p, bool force) {
  if (p.bits != 4 || p.M > 16 || p.K % wm::kUnitK != 0 || p.N % kTileN != 0) return false;
  if (!force && p.M > 8 && static_cast<long>(p.N / kTileN) * (p.K / wm::kUnitK) < 4096) return false;
  if (p.group_size < p.K) {                  // a unit lies in one group, whose index is a shift of the unit's
    bool ok = false;
    for (int s = 0; s < 24; ++s) ok = ok || (wm::kUnitK << s) == p.group_size;
    if (!ok) return false;
  }
  const uintptr_t low = reinterpret_cast<uintptr_t>(p.bp) | reinterpret_cast<uintptr_t>(p.scales) |
                        reinterpret_cast<uintptr_t>(p.qzeros) | reinterpret_cast<uintptr_t>(p.a) |
                        reinterpret_cast<uintptr_t>(p.workspace);
  if (low & 15) return false;                // 16-byte copies
  // pairs of fp16 (the tile-split kernel's unsplit form goes by single values; fused operands lie on 8 bytes for every kernel)
  if ((reinterpret_cast<uintptr_t>(p.bias) | reinterpret_cast<uintptr_t>(p.c)) & 3) return false;
  if (p.epilogue == B200_EPI_SILU_MUL && ((p.N / kTileN) & 1)) return false;
  if (p.epilogue == kEpiRopeKv && p.fe && !(p.fe->D == 32 || p.fe->D == 64 || p.fe->D == 128)) return false;
  UnitCut cut;
  return (p.M <= 8 ? wm::cut_of<1>(p, cut) : wm::cut_of<2>(p, cut)) > 0;
}

bool launch_wna16_mma(const WnaParams& p, cudaStream_t st, bool force) {
  if (!wna16_mma_takes(p, force)) return false;
  return p.M <= 8 ? wm::launch_nt<1>(p, st) : wm::launch_nt<2>(p, st);
}

}  // namespace b200
