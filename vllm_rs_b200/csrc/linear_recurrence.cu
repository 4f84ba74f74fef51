// Recurrent sequence mixers with a per-sequence state slot, for ragged steps (a prompt portion of any length or one
// decoded token per sequence): the short causal convolution in front of them, the gated delta rule, and the
// scalar-decay state-space scan (SSD form of Mamba-2).  State lives in fp32 in slot-indexed pools owned by the caller;
// a sequence that starts at position 0 in this step (context == rows of the step) starts from zeros whatever its
// slot held before, so slots can be handed on without clearing.  Everything here is fp32.
//
//   short_conv_silu : y[t, c] = silu(bias[c] + sum_j w[c, j] * x[t - (taps-1) + j, c]); the last taps-1 inputs of a
//                     sequence are its conv state  [slots, taps-1, C].  Token chunks run in parallel; a second small
//                     launch rolls the state forward.
//   delta_rule      : per head, S [dim, vdim]:  S <- g S;  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q
//                     with q, k unit-normalised per head (q also times dim^-1/2), beta = sigmoid(b),
//                     g = exp(-exp(a_log) * softplus(a + dt_bias)).  state [slots, heads, dim, vdim].  In the
//                     channel form g is one decay per head AND key channel (row i of S is multiplied by g[i]), handed
//                     in ready-made (lowrank_decay kind 1 makes it from a low-rank projection).
//   ssd_scan        : per head, S [nstate, vdim]:  dt = softplus(dt_raw + dt_bias);  S <- exp(-exp(a_log) dt) S + dt B x^T;
//                     y = S^T C + D x.  state [slots, heads, nstate, vdim].
//   decay_attn      : per head, S [dim, vdim]:  S <- diag(a_t) S + k_t v_t^T;  o_t = S^T q_t  (linear attention with a decayed
//                     state, no softmax or denominator).  a_t is one constant per head (retention-style fixed decays) or
//                     one value per key channel and token (gated linear attention; lowrank_decay makes it from a
//                     low-rank projection: sigmoid(z)^(1/tau)).  Optional SiLU on q, k, v and scales on q and k.
//                     state [slots, heads, dim, vdim].
// The three scans share two kernels.  scan_short_kernel takes the sequences that bring few tokens, one after another.  scan_kernel
// walks longer portions
// in blocks of eight tokens, within which the recurrence is unrolled exactly: with G_t the product of the block's decays up to
// token t and S0 the state before it,
//   k_t^T S_(t-1) = G_t k_t^T S0 + sum_(j<t) (G_t / G_j) (k_t . k_j) u_j,   S_t^T q_t likewise,   S_8 = G_8 S0 + sum_j (G_8 / G_j) k_j u_j^T
// so that the eight tokens' products with the state are independent of each other and their sums over the lanes meet in one
// exchange; the u_t follow from a product with the inverse of an 8 x 8 unit triangle.  Decay ratios are products of decays,
// never quotients.  All fp32.
#include "../../include/b200_vllm.h"
#include <algorithm>
#include <type_traits>

#include "f32x2.cuh"
#include "seqmix.cuh"

namespace b200 {
using namespace seqmix;

constexpr int kMaxTaps = 8;

constexpr int kConvChunk = 64;      // tokens per thread

// grid = (channel blocks, sequences, token chunks): every thread convolves one channel over one chunk of a sequence's
// rows; the taps-1 inputs before the chunk come from the rows before it or, at the start of the step, from the
// sequence's state (zeros when the sequence starts here).  out must not alias x.
template <int TAPS>
__global__ void short_conv_silu_kernel(float* __restrict__ out, int ldo, const float* __restrict__ x, int ldx,
                                       const float* __restrict__ taps_w, const float* __restrict__ bias,
                                       const float* __restrict__ state, const int32_t* __restrict__ slots,
                                       const uint32_t* __restrict__ cu, const uint32_t* __restrict__ ctx, int C) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y;
  if (c >= C) return;
  const int t0 = cu[b], t1 = cu[b + 1];
  const int start = t0 + static_cast<int>(blockIdx.z) * kConvChunk;
  if (start >= t1) return;
  const int end = min(t1, start + kConvChunk);
  const bool fresh = static_cast<int>(ctx[b]) == t1 - t0;
  constexpr int P = TAPS - 1;                  // inputs remembered between tokens
  float w[TAPS], win[P > 0 ? P : 1];
#pragma unroll
  for (int j = 0; j < TAPS; ++j) w[j] = taps_w[static_cast<size_t>(c) * TAPS + j];
  const float* sp = state + static_cast<size_t>(slots[b]) * P * C + c;
#pragma unroll
  for (int j = 0; j < P; ++j) {                // oldest first
    const int idx = start - P + j;
    win[j] = idx >= t0 ? x[static_cast<size_t>(idx) * ldx + c] : (fresh ? 0.f : sp[static_cast<size_t>(P + idx - t0) * C]);
  }
  const float bv = bias ? bias[c] : 0.f;
  for (int t = start; t < end; ++t) {
    const float xv = x[static_cast<size_t>(t) * ldx + c];
    float acc = bv;
#pragma unroll
    for (int j = 0; j < P; ++j) acc += w[j] * win[j];
    acc += w[P] * xv;
    out[static_cast<size_t>(t) * ldo + c] = silu_exact(acc);
#pragma unroll
    for (int j = 0; j + 1 < P; ++j) win[j] = win[j + 1];
    if (P > 0) win[P > 0 ? P - 1 : 0] = xv;
  }
}

// the sequence's last taps-1 inputs become its state (older ones slide over from the previous state)
template <int TAPS>
__global__ void short_conv_state_kernel(const float* __restrict__ x, int ldx, float* __restrict__ state,
                                        const int32_t* __restrict__ slots, const uint32_t* __restrict__ cu,
                                        const uint32_t* __restrict__ ctx, int C) {
  constexpr int P = TAPS - 1;
  const int c = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y;
  if (c >= C || P == 0) return;
  const int t0 = cu[b], t1 = cu[b + 1];
  if (t1 <= t0) return;
  const bool fresh = static_cast<int>(ctx[b]) == t1 - t0;
  float* sp = state + static_cast<size_t>(slots[b]) * P * C + c;
  float keep[P > 0 ? P : 1];
#pragma unroll
  for (int j = 0; j < P; ++j) {
    const int idx = t1 - P + j;
    keep[j] = idx >= t0 ? x[static_cast<size_t>(idx) * ldx + c] : (fresh ? 0.f : sp[static_cast<size_t>(P + idx - t0) * C]);
  }
#pragma unroll
  for (int j = 0; j < P; ++j) sp[static_cast<size_t>(j) * C] = keep[j];
}

__device__ __forceinline__ void cp_async4(float* smem, const float* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(smem))),
               "l"(gmem)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async16(float* smem, const float* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(smem))),
               "l"(gmem)
               : "memory");
}
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ float sum2(f2 v) {
  float lo, hi;
  unpack2(v, lo, hi);
  return lo + hi;
}

constexpr int kOneCols = 16;                   // columns of S per block of threads: single tokens
constexpr int kBT = 8;                         // tokens per block of the recurrence
constexpr int kRing = 8;                       // blocks of tokens in shared memory (sixteen are no faster)
constexpr int kSorted = 64;                    // sequences up to which a step's longest go first
constexpr int kShort = 16;                     // tokens of a sequence up to which it is walked token by token
constexpr int kDelta = 0, kDecay = 1, kSsd = 2;

using ScanArgs = b200_scan_args;

constexpr int CW = 4;                          // columns of the state per walking warp
template <int DK, bool CHAN, int WW> struct ScanSmem {         // WW: walking warps
  static constexpr int kRows = kBT * DK;                                        // floats of one array of token rows
  static constexpr int kG = (CHAN ? 3 : 2) * kRows;                             // k | q | decays | scalars | T, P (8 x 8 each) | ..
  static constexpr int kCols = WW * CW, kMat = kG + 4 * kBT;                 // rest of G_7, strength, G_t, W_t per token
  static constexpr int kRat = kMat + 2 * kBT * kBT;                             // [t][j] decay from token j to token t
  static constexpr int kGend = kRat + kBT * kBT;                                // CHAN: [DK] decays over the block, [DK] their rests
  static constexpr int kGrest = kGend + (CHAN ? DK : 0), kBuf = kGrest + (CHAN ? DK : 0);
  static constexpr int kU = kRing * kBuf;                                       // [WW][8 tokens][4 columns]
  static constexpr int kBars = kU + WW * kBT * CW;
  static constexpr int kBytes = kBars * 4 + 2 * kRing * 8 + 16;
};
// CH floats from shared memory
template <int CH> __device__ __forceinline__ void ldv(float (&x)[CH], const float* p) {
  if constexpr (CH % 4 == 0) {
#pragma unroll
    for (int i = 0; i < CH; i += 4) {
      const float4 v = *reinterpret_cast<const float4*>(p + i);
      x[i] = v.x; x[i + 1] = v.y; x[i + 2] = v.z; x[i + 3] = v.w;
    }
  } else {
    const float2 v = *reinterpret_cast<const float2*>(p);
    x[0] = v.x; x[1] = v.y;
  }
}
template <int CH> __device__ __forceinline__ void stv(float* p, const float (&x)[CH]) {
  if constexpr (CH % 4 == 0) {
#pragma unroll
    for (int i = 0; i < CH; i += 4) *reinterpret_cast<float4*>(p + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
  } else {
    *reinterpret_cast<float2*>(p) = make_float2(x[0], x[1]);
  }
}
template <int CH> __device__ __forceinline__ void ldv2(f2 (&x)[CH / 2], const float* p) {
  if constexpr (CH % 4 == 0) {
#pragma unroll
    for (int i = 0; i < CH; i += 4) {
      const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p + i);
      x[i / 2] = v.x; x[i / 2 + 1] = v.y;
    }
  } else {
    x[0] = *reinterpret_cast<const f2*>(p);
  }
}
// 32 values per lane -> lane l holds the sum over the lanes of value l: a butterfly that halves the values
__device__ __forceinline__ float meet32(float (&x)[32], int lane) {
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) {
    const bool up = lane & w;
#pragma unroll
    for (int i = 0; i < w; ++i) {
      const float keep = up ? x[i + w] : x[i], send = up ? x[i] : x[i + w];
      x[i] = keep + __shfl_xor_sync(0xffffffffu, send, w);
    }
  }
  return x[0];
}
// The same where lane l has the values of token t (of eight, four columns each) at t ^ (l >> 2): what a lane keeps in the first three
// exchanges is always the first half, and nothing has to be selected.
__device__ __forceinline__ float meet32_turned(float (&x)[32], int lane) {
#pragma unroll
  for (int w = 16; w > 2; w >>= 1)
#pragma unroll
    for (int i = 0; i < w; ++i) x[i] += __shfl_xor_sync(0xffffffffu, x[i + w], w);
#pragma unroll
  for (int w = 2; w > 0; w >>= 1) {
    const bool up = lane & w;
#pragma unroll
    for (int i = 0; i < w; ++i) {
      const float keep = up ? x[i + w] : x[i], send = up ? x[i] : x[i + w];
      x[i] = keep + __shfl_xor_sync(0xffffffffu, send, w);
    }
  }
  return x[0];
}
// The walkers of a whole cluster arrive on the preparing block's barrier.
__device__ __forceinline__ bool wait_cluster(uint64_t* bar, uint32_t parity, volatile int* fail, int* err) {
  const uint32_t at = smem_u32(bar);
#pragma unroll 1
  for (int i = 0;; ++i) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred P;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P, [%1], %2;\n\tselp.u32 %0, 1, 0, P;\n\t}"
                 : "=r"(ok) : "r"(at), "r"(parity) : "memory");
    if (ok) return true;
    if (*fail || i > (1 << 24)) {
      *reinterpret_cast<volatile int*>(err) = 1;
      *fail = 1;
      return false;
    }
  }
}

// Portions of more than `above` tokens, up to `to`.  grid = (column blocks, heads, runs of sequences); a block walks its sequences one after
// another.  The first WW warps each own four columns of S: a lane holds DK / 32 neighbouring rows of them in registers, so that
// a key or query row is read once from shared memory for four columns (one column per lane made these reads the bound: 512
// bytes of registers per load and warp).  Two groups of four warps prepare blocks of tokens under the walks of the blocks before: rows read a
// turn ahead into registers, normed or activated, and the block's triangles.  What they prepare is the same for all columns of a head, so
// nc neighbouring blocks form a cluster, take turns at it and send it to each other's rings by bulk copies: prepared eight
// times over, in each of the blocks of a head of 128 columns, it took issue slots from the walk (4096 tokens of 16 heads of 128 x 128:
// 597 us, 423 for the walk alone).
// WW = 8 lets two walking warps share a scheduler and a prepared block, WW = 4 spreads few columns over more SMs.
// Bound: the chain of blocks, one walk after another; a walk's 78 shuffles (6.3 cycles each from one warp of a scheduler), its 16-byte loads
// (12) and its packed FMAs (2.7) overlap in part.  HBM and the FMA units would take 16 and 89 us for 4096 tokens of 16 heads of
// 128 x 128.  Measured there, token by token (eight lanes per column, four chained shuffles per token) -> in blocks -> prepared in turns,
// and sums that meet without selections (meet32_turned: 510 -> 440): delta rule 2278 -> 597 -> 445 us; decayed state of 8 heads of
// 128 x 256: 909 -> 398 -> 337 us.  Two columns per warp and twice the warps: slower (shared memory's loads per column double).  The
// state's update does not wait for the read-out's sums: the queries' products are taken before the correction's sums meet, and
// meet under the update (665 and 424 us with both in turn).
template <int DK, int MODE, bool CHAN, int WW>
__global__ void __launch_bounds__(WW * 32 + 256, 1)
scan_kernel(const ScanArgs a, int num_seqs, int above, int to, int nc, int* err) {
  using SM = ScanSmem<DK, CHAN, WW>;
  constexpr int CH = DK / 32, COLS = SM::kCols;
  constexpr bool BACK = MODE != kDelta || WW == 8;                     // rows of the triangles from the diagonal back (below)
  extern __shared__ __align__(16) float sm[];
  uint64_t* ready = reinterpret_cast<uint64_t*>(sm + SM::kBars);
  uint64_t* done = ready + kRing;
  volatile int* fail = reinterpret_cast<volatile int*>(done + kRing);
  const int h = blockIdx.y, tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31, col0 = blockIdx.x * COLS;
  const int rank = nc > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int dim = a.dim, vdim = a.vdim, hk = MODE == kDecay ? h : h / (a.heads / a.kv_heads);
  constexpr int kAll = WW * 32 + 256;
  if (above > kShort) pdl_trigger();                                   // the launch for shorter sequences follows
  // Longest sequences first: where not all blocks fit the chip at once, the last to start have the least to do.  Three sequences
  // of 500, 1000 and 1501 tokens, 8 heads of 128 x 256 (192 blocks): 2001 tokens in a row before, 1501 now; the four scans of a
  // hybrid step take 960 us instead of 1256.  One sequence has no order to look up.
  __shared__ uint8_t order[kSorted];
  const bool sorted = num_seqs > 1 && num_seqs <= kSorted;
  if (sorted && tid < num_seqs) {
    const uint32_t n = a.cu_seqlens_q[tid + 1] - a.cu_seqlens_q[tid];
    int rank = 0;
    for (int i = 0; i < num_seqs; ++i) {
      const uint32_t m = a.cu_seqlens_q[i + 1] - a.cu_seqlens_q[i];
      rank += m > n || (m == n && i < tid);
    }
    order[rank] = static_cast<uint8_t>(tid);
  }
  __syncthreads();
  auto of_this = [&](int tokens) { return tokens > above && tokens <= to; };
  auto seq = [&](int z) { return sorted ? static_cast<int>(order[z]) : z; };
  {
    int mine = 0;                                                      // a sequence for this kernel among the block's
    for (int z = blockIdx.z + tid * gridDim.z; z < num_seqs; z += kAll * gridDim.z)
      mine |= of_this(static_cast<int>(a.cu_seqlens_q[seq(z) + 1] - a.cu_seqlens_q[seq(z)]));
    if (!__syncthreads_or(mine)) {
      pdl_wait();
      return;
    }
  }
  if (tid == 0) {
    for (int i = 0; i < kRing; ++i) { mbar_init(&ready[i], 4); mbar_init(&done[i], WW * nc); }
    *fail = 0;
    fence_barrier_init();
  }
  // what no token writes is zero and stays it: the triangles' upper halves
  for (int e = tid; e < kRing * 2 * kBT * kBT; e += kAll) sm[e / (2 * kBT * kBT) * SM::kBuf + SM::kMat + e % (2 * kBT * kBT)] = 0.f;
  fence_proxy_async();                                                 // before the bulk copies that other blocks send there
  __syncthreads();
  if (nc > 1) {                                                        // the others' barriers are there
    cluster_arrive();
    cluster_wait();
  }
  int blocks = 0;                                                      // blocks of tokens so far, over all sequences
  for (int z = blockIdx.z; z < num_seqs; z += gridDim.z) {
    const int b = seq(z), t0 = a.cu_seqlens_q[b], t1 = a.cu_seqlens_q[b + 1], nblk = (t1 - t0 + kBT - 1) / kBT;
    if (!of_this(t1 - t0)) continue;                                   // (another launch's)
    const bool fresh = static_cast<int>(a.context_lens[b]) == t1 - t0;
    if (warp >= WW) {
      // ---------------------------------------------------------- token rows
      const int pt = tid & 127, pw = warp & 3, grp = (warp - WW) >> 2;
      const bool wide = dim % 4 == 0 && (a.ld_q | a.ld_k) % 4 == 0 && (!CHAN || a.ld_decay % 4 == 0) &&
                        ((reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.k) |
                          (CHAN ? reinterpret_cast<uintptr_t>(a.chan_decay) : 0)) & 15) == 0;
      // A block of tokens is prepared by one group of one block of the cluster, g being its number over all sequences, in the order of the
      // ring's places; its rows are read a turn ahead into registers.
      const int step = 2 * nc, first = (grp * nc + rank - blocks) & (step - 1);
      constexpr int TPR = DK / 4, RPS = 128 / TPR, NR = kBT / RPS;     // threads per row, rows at a time, rows of a thread
      // (rows of 256 entries do not fit beside the triangles' operands but where there are fewer threads and triangles)
      constexpr bool kAhead = DK <= 128 || (MODE != kDelta && !CHAN && WW == 4);
      float4 raw_k[NR], raw_q[NR], raw_d[CHAN ? NR : 1];
      const int rx = pt % TPR * 4;
      auto read_rows = [&](int i) {
        const int c0 = t0 + i * kBT;
#pragma unroll
        for (int z = 0; z < NR; ++z) {
          const int t = c0 + pt / TPR + z * RPS;
          const bool in = i < nblk && t < t1 && rx < dim;
          auto get = [&](const float* p) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (in && wide) {
              v = __ldg(reinterpret_cast<const float4*>(p));
            } else if (in) {
              v.x = __ldg(p);
              if (rx + 1 < dim) v.y = __ldg(p + 1);
              if (rx + 2 < dim) v.z = __ldg(p + 2);
              if (rx + 3 < dim) v.w = __ldg(p + 3);
            }
            return v;
          };
          raw_k[z] = get(a.k + static_cast<size_t>(t) * a.ld_k + hk * dim + rx);
          raw_q[z] = get(a.q + static_cast<size_t>(t) * a.ld_q + hk * dim + rx);
          if (CHAN) raw_d[z] = get(a.chan_decay + static_cast<size_t>(t) * a.ld_decay + h * dim + rx);
        }
      };
      auto sync = [&] {                                // of these four warps
        __syncwarp();
        asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory");
      };
      const float neg_a = MODE == kDecay || CHAN ? 0.f : -expf(a.a_log[h]), dtb = MODE == kDecay || CHAN ? 0.f : a.dt_bias[h];
      const float hd = MODE == kDecay && !CHAN ? a.head_decay[h] : 1.f;
      const float qn = rsqrtf(static_cast<float>(dim));
      // The scalars of a block, by the group's last warp, a block ahead: raw values in registers, then decays, strengths, products.
      float raw_b = 0.f, raw_a = 0.f;
      auto read_scalars = [&](int i) {
        const int t = t0 + i * kBT + lane;
        if (lane >= kBT || t >= t1) return;
        const size_t o = static_cast<size_t>(t) * a.ld_s + h;
        if (MODE == kDelta) raw_b = a.strength[o];
        if (MODE == kSsd || (MODE == kDelta && !CHAN)) raw_a = a.decay_raw[o];
      };
      auto make_scalars = [&](int i) {
        float* G = sm + (blocks + i) % kRing * SM::kBuf + SM::kG;
        float g = 1.f, w = 0.f;                        // decay; write strength
        if (lane < kBT && t0 + i * kBT + lane < t1) {
          if (MODE == kDelta) {
            w = sigmoid_f(raw_b);
            if (!CHAN) g = expf(neg_a * softplus_f(raw_a + dtb));
          } else if (MODE == kSsd) {
            w = softplus_f(raw_a + dtb);
            g = expf(neg_a * w);
          } else {
            w = a.k_scale;
            g = hd;
          }
        }
        // decay from token j to token t: the products g_(j+1) .. g_t; from the block's start, and to its end
        float* R = G + (SM::kRat - SM::kG);
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          const int t = (lane >> 3) + z * 4, j = lane & 7;
          float r = 1.f, rest = 0.f;                   // the product and what its roundings left
          auto times = [&](float x) {
            const float p = __fmul_rn(r, x);
            if (MODE == kDecay) rest = fmaf(rest, x, fmaf(r, x, -p));
            r = p;
          };
#pragma unroll
          for (int m = 1; m < kBT; ++m) {
            const float gm = __shfl_sync(0xffffffffu, g, m);
            if (m > j && m <= t) times(gm);
          }
          R[t * kBT + j] = r + rest;
          if (t == kBT - 1) G[3 * kBT + j] = r + rest;
          const float g0 = __shfl_sync(0xffffffffu, g, 0);
          if (j == 0) {
            times(g0);
            const float whole = r + rest;
            G[2 * kBT + t] = whole;
            if (t == kBT - 1) G[0] = rest - (whole - r);
          }
        }
        if (lane < kBT) G[kBT + lane] = w;
      };
      // which entry of a triangle, row after row, this lane gets: M (rows 1 .., j < t) for warp 1, P (j <= t) from row 4 on for warp
      // 0, of rows 0 - 3 for warp 2
      int et = pw == 1 ? 1 : pw == 0 ? 4 : 0, ej = lane;
      const int et_end = pw == 2 ? 4 : kBT;
      while (et < et_end && ej >= (pw == 1 ? et : et + 1)) {
        ej -= pw == 1 ? et : et + 1;
        ++et;
      }
      if (kAhead) read_rows(first);
      if (pw == 3) read_scalars(first);
      for (int i = first; i < nblk; i += step) {
        const int g = blocks + i, n = min(kBT, t1 - t0 - i * kBT);
        float* B = sm + g % kRing * SM::kBuf;
        const float* G = B + SM::kG;
        if (!kAhead) read_rows(i);
        if (g >= kRing) wait_cluster(&done[g % kRing], (g / kRing - 1) & 1, fail, err);
        __syncwarp();
#pragma unroll
        for (int z = 0; z < NR; ++z) {
          float* row = B + (pt / TPR + z * RPS) * DK + rx;
          *reinterpret_cast<float4*>(row) = raw_k[z];
          *reinterpret_cast<float4*>(row + SM::kRows) = raw_q[z];
          if (CHAN) *reinterpret_cast<float4*>(row + 2 * SM::kRows) = raw_d[z];
        }
        if (kAhead) read_rows(i + step);
        sync();
        // ---- two tokens per warp: norms or activation, in place; past the end: no key, no value, decay one
        if (MODE == kDelta || (MODE == kDecay && a.act) || n < kBT) {
          float kx[2][CH], qx[2][CH], sk[2] = {0.f, 0.f}, sq[2] = {0.f, 0.f};
          float* kr = B + pw * 2 * DK + lane * CH;
#pragma unroll
          for (int z = 0; z < 2; ++z) {
            ldv<CH>(kx[z], kr + z * DK);
            ldv<CH>(qx[z], kr + SM::kRows + z * DK);
#pragma unroll
            for (int j = 0; j < CH; ++j) {
              if (MODE == kDelta) {
                sk[z] += kx[z][j] * kx[z][j];
                sq[z] += qx[z][j] * qx[z][j];
              } else if (MODE == kDecay && a.act) {
                kx[z][j] = silu_exact(kx[z][j]);
                qx[z][j] = silu_exact(qx[z][j]);
              }
            }
          }
          float ik[2] = {1.f, 1.f}, iq[2] = {1.f, 1.f};
          if (MODE == kDelta) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
              for (int z = 0; z < 2; ++z) {
                sk[z] += __shfl_xor_sync(0xffffffffu, sk[z], o);
                sq[z] += __shfl_xor_sync(0xffffffffu, sq[z], o);
              }
#pragma unroll
            for (int z = 0; z < 2; ++z) {
              ik[z] = 1.f / sqrtf(sk[z] + 1e-6f);
              iq[z] = qn / sqrtf(sq[z] + 1e-6f);
            }
          }
#pragma unroll
          for (int z = 0; z < 2; ++z) {
            const int r = pw * 2 + z;
            const bool in = r < n;
#pragma unroll
            for (int j = 0; j < CH; ++j) {
              kx[z][j] = in ? kx[z][j] * ik[z] : 0.f;
              qx[z][j] = in ? qx[z][j] * iq[z] : 0.f;
            }
            stv<CH>(kr + z * DK, kx[z]);
            stv<CH>(kr + SM::kRows + z * DK, qx[z]);
            if (CHAN && !in) {
#pragma unroll
              for (int j = 0; j < CH; ++j) kx[z][j] = 1.f;
              stv<CH>(kr + 2 * SM::kRows + z * DK, kx[z]);
            }
          }
        }
        sync();
        // ---- P (t, j) = decayed q_t . k_j, j <= t, and (delta) M (t, j) = beta_t times the decayed k_t . k_j, j < t, then
        // T = (1 + M)^-1.  A lane holds its rows of all eight tokens; the sums over the lanes go an entry to a lane.
        // A walking lane must not meet a later token's part, which may be infinite or NaN and reach back through its zero of the
        // triangle; in its place it takes its own.  BACK: rows are stored from the diagonal back (entry d: token t - d, zero past
        // the first), and a shuffle from d tokens below gives a lane's own part where there is none.  Otherwise as they are, with
        // the source lanes in registers, which eight walking warps do not have.  Delta rule, 4096 tokens of heads of 128 x 128:
        // 16 heads 650 us with BACK, 590 without (a branch instead: 666); 32 heads, a decay per channel 907 - 965 and 1114.
        // Decayed state, 8 heads of 128 x 256: 384 and 397.
        float v = 0.f;
        if (pw == 3) {
          make_scalars(i);
          read_scalars(i + step);
        } else if (pw != 1 || MODE == kDelta) {
          auto entries = [&](auto first, auto last, auto strict, const float* rows) {
            constexpr int F = decltype(first)::value, L = decltype(last)::value, ST = decltype(strict)::value;
            float y[kBT][CH], x[32];
#pragma unroll
            for (int e = 0; e < 32; ++e) x[e] = 0.f;
            int e = 0;
#pragma unroll
            for (int t = 0; t < L; ++t) {
              ldv<CH>(y[t], B + t * DK + lane * CH);
              if (CHAN) {                              // y[j] becomes k_j decayed up to token t
                float dt[CH];
                ldv<CH>(dt, B + 2 * SM::kRows + t * DK + lane * CH);
#pragma unroll
                for (int j = 0; j < t; ++j)
#pragma unroll
                  for (int c = 0; c < CH; ++c) y[j][c] *= dt[c];
              }
              if (t < F) continue;
              float xt[CH];
              ldv<CH>(xt, rows + t * DK + lane * CH);
#pragma unroll
              for (int j = 0; j <= t - ST; ++j) {
                float acc = xt[0] * y[j][0];
#pragma unroll
                for (int c = 1; c < CH; ++c) acc += xt[c] * y[j][c];
                x[e++] = acc;
              }
            }
            return meet32(x, lane);
          };
          using std::integral_constant;
          const float* K = B;
          const float* Q = B + SM::kRows;
          v = pw == 1   ? entries(integral_constant<int, 1>{}, integral_constant<int, kBT>{}, integral_constant<int, 1>{}, K)
                    : pw == 0 ? entries(integral_constant<int, 4>{}, integral_constant<int, kBT>{}, integral_constant<int, 0>{}, Q)
                              : entries(integral_constant<int, 0>{}, integral_constant<int, 4>{}, integral_constant<int, 0>{}, Q);
        }
        sync();
        if (pw != 3 && (pw != 1 || MODE == kDelta)) {
          float* out = B + SM::kMat + (pw == 1 ? 0 : kBT * kBT);
          if (et < et_end) {
            v *= B[SM::kRat + et * kBT + ej];
            out[et * kBT + (pw != 1 && BACK ? et - ej : ej)] = pw == 1 ? v * G[kBT + et] : v;
          }
          if (pw == 1) {                               // column `lane` of T by forward substitution
            __syncwarp();
            float tc[kBT];
#pragma unroll
            for (int t = 0; t < kBT; ++t) {
              const float4 ma = *reinterpret_cast<const float4*>(out + t * kBT), mb = *reinterpret_cast<const float4*>(out + t * kBT + 4);
              const float m[kBT] = {ma.x, ma.y, ma.z, ma.w, mb.x, mb.y, mb.z, mb.w};
              float acc = t == lane ? 1.f : 0.f;
#pragma unroll
              for (int j = 0; j < t; ++j) acc -= m[j] * tc[j];
              tc[t] = acc;
            }
            __syncwarp();
            if (lane < kBT) {
#pragma unroll
              for (int t = 0; t < kBT; ++t) out[t * kBT + (BACK ? (t - lane) & (kBT - 1) : lane)] = tc[t];
            }
          }
        }
        if (CHAN) {
          // k <- G_t k_t, q <- G_t q_t, decays <- W_t k_t, per channel; the block's whole decay
          sync();
          for (int e = pt; e < DK; e += 128) {
            float kr[kBT], d[kBT], g = 1.f, rest = 0.f;
#pragma unroll
            for (int t = 0; t < kBT; ++t) {
              kr[t] = B[t * DK + e];
              d[t] = e < dim ? B[2 * SM::kRows + t * DK + e] : 1.f;
              if (MODE == kDecay) {                    // (with what the products' roundings leave)
                const float p = __fmul_rn(g, d[t]);
                rest = fmaf(rest, d[t], fmaf(g, d[t], -p));
                g = p;
              } else {
                g *= d[t];
              }
              B[t * DK + e] = kr[t] * g;
              B[SM::kRows + t * DK + e] *= g;
            }
            if (MODE == kDecay) {
              const float whole = g + rest;
              B[SM::kGrest + e] = rest - (whole - g);
              g = whole;
            }
            B[SM::kGend + e] = g;
            g = 1.f;
#pragma unroll
            for (int t = kBT - 1; t >= 0; --t) {
              B[2 * SM::kRows + t * DK + e] = kr[t] * g;
              g *= d[t];
            }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&ready[g % kRing]);
        if (nc > 1) {                                  // to the same place of the cluster's other blocks
          fence_proxy_async();
          sync();
          if (pw == 0 && lane < nc && lane != rank && !*fail)          // (after a wait gave up, nothing more is sent)
            asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                             mapa_shared(smem_u32(B), lane)),
                         "r"(smem_u32(B)), "r"(SM::kBuf * 4), "r"(mapa_shared(smem_u32(&ready[g % kRing]), lane))
                         : "memory");
        }
      }
    } else {
      // ---------------------------------------------------------- the walk
      const int colw = col0 + warp * CW;               // this warp's first column
      float* sp = a.state + ((static_cast<size_t>(a.state_slots[b]) * a.heads + h) * dim) * vdim + colw;
      const bool wide_s = vdim % 4 == 0 && (reinterpret_cast<uintptr_t>(a.state) & 15) == 0;
      const float skip = MODE == kSsd && a.d_skip ? a.d_skip[h] : 0.f;
      f2 s[CW][CH / 2];                                // [column][pair of rows]
      {
        float x[CH][CW];
#pragma unroll
        for (int r = 0; r < CH; ++r) {
          const int i = lane * CH + r;
#pragma unroll
          for (int c = 0; c < CW; ++c) x[r][c] = 0.f;
          if (!fresh && i < dim) {
            const float* src = sp + static_cast<size_t>(i) * vdim;
            if (wide_s && colw < vdim) {
              ldv<CW>(x[r], src);
            } else {
#pragma unroll
              for (int c = 0; c < CW; ++c)
                if (colw + c < vdim) x[r][c] = src[c];
            }
          }
        }
#pragma unroll
        for (int c = 0; c < CW; ++c)
#pragma unroll
          for (int r = 0; r < CH; r += 2) s[c][r / 2] = pack2(x[r][c], x[r + 1][c]);
      }
      float* us = sm + SM::kU + warp * kBT * CW;
      const int tt = lane >> 2, cc = lane & 3;         // the token and column whose sums this lane gets
      int from[kBT];
#pragma unroll
      for (int j = 0; j < kBT; ++j) from[j] = min(j, tt) * 4 + cc;
      // its values, two blocks ahead
      const bool col_in = colw + cc < vdim;
      const float* vp = a.v + static_cast<size_t>(t0 + tt) * a.ld_v + h * vdim + colw + cc;
      const size_t v_step = static_cast<size_t>(kBT) * a.ld_v;
      int v_left = col_in ? (t1 - t0 - tt + kBT - 1) / kBT : 0;        // blocks in which this lane has a token
      auto value = [&] {
        const float v = v_left > 0 ? __ldg(vp) : 0.f;
        vp += v_step;
        --v_left;
        return v;
      };
      float v0 = value(), v1 = value();
      float* op = a.out + (static_cast<size_t>(t0 + tt) * a.heads + h) * vdim + colw + cc;
      const size_t o_step = static_cast<size_t>(kBT) * a.heads * vdim;
      // A block that another one prepares arrives by its bytes; who waits for them says so, a block ahead.
      auto expect = [&](int g) {
        if (nc > 1 && warp == 0 && lane == 0 && (g & (nc - 1)) != rank) {
          const uint32_t bar = smem_u32(&ready[g % kRing]);
          asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(SM::kBuf * 4) : "memory");
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], 4;" ::"r"(bar) : "memory");
        }
      };
      expect(blocks);
      // what entry j of a row of the triangles is multiplied by; the oldest token first in both forms, so that their bits are equal
      auto entry = [](int i) { return BACK ? kBT - 1 - i : i; };
      auto part = [&](float x, int j) { return BACK ? __shfl_up_sync(0xffffffffu, x, j * 4) : __shfl_sync(0xffffffffu, x, from[j]); };
      for (int i = 0; i < nblk; ++i) {
        const int g = blocks + i;
        if (i + 1 < nblk) expect(g + 1);
        float vt = v0;
        v0 = v1;
        const bool has = v_left > -2;                  // (of the block at hand)
        v1 = value();
        mbar_wait_limited(&ready[g % kRing], (g / kRing) & 1, fail, err);
        __syncwarp();
        const float* B = sm + g % kRing * SM::kBuf;
        const float* G = B + SM::kG;
        // the rows' products with this lane's part of the state
        constexpr bool KEEP = MODE == kDelta && !CHAN && WW == 4 && DK <= 128;     // keys stay in registers until the update
        f2 kept[KEEP ? kBT : 1][CH / 2];
        auto dots = [&](float (&x)[32], const float* rows, auto keep) {
#pragma unroll
          for (int t = 0; t < kBT; ++t) {
            f2 y[CH / 2];
            ldv2<CH>(y, rows + (decltype(keep)::value ? t : t ^ tt) * DK + lane * CH);
            if (decltype(keep)::value) {
#pragma unroll
              for (int r = 0; r < CH / 2; ++r) kept[KEEP ? t : 0][r] = y[r];
            }
#pragma unroll
            for (int c = 0; c < CW; ++c) {
              f2 acc = mul2(y[0], s[c][0]);
#pragma unroll
              for (int r = 1; r < CH / 2; ++r) acc = fma2(y[r], s[c][r], acc);
              x[t * CW + c] = sum2(acc);
            }
          }
        };
        const float gt = CHAN ? 1.f : G[2 * kBT + tt];
        const float wt = G[kBT + tt];
        if (MODE == kDecay && a.act) vt = silu_exact(vt);
        float u = vt * wt, xq[32];
        dots(xq, B + SM::kRows, std::false_type{});
        if (MODE == kDelta) {
          float xk[32];
          dots(xk, B, std::integral_constant<bool, KEEP>{});
          const float r = wt * fmaf(-gt, KEEP ? meet32(xk, lane) : meet32_turned(xk, lane), vt);
          const float4 ta = *reinterpret_cast<const float4*>(B + SM::kMat + tt * kBT), tb = *reinterpret_cast<const float4*>(B + SM::kMat + tt * kBT + 4);
          const float T[kBT] = {ta.x, ta.y, ta.z, ta.w, tb.x, tb.y, tb.z, tb.w};
          u = 0.f;
#pragma unroll
          for (int z = 0; z < kBT; ++z) u = fmaf(T[entry(z)], part(r, entry(z)), u);
        }
        us[lane] = CHAN ? u : u * G[3 * kBT + tt];
        __syncwarp();
        const float e = meet32_turned(xq, lane);              // (in no one's way: the state's update does not need it)
        {
          const float4 pa = *reinterpret_cast<const float4*>(B + SM::kMat + kBT * kBT + tt * kBT);
          const float4 pb = *reinterpret_cast<const float4*>(B + SM::kMat + kBT * kBT + tt * kBT + 4);
          const float P[kBT] = {pa.x, pa.y, pa.z, pa.w, pb.x, pb.y, pb.z, pb.w};
          float o = __fmul_rn(gt, e);
#pragma unroll
          for (int z = 0; z < kBT; ++z) o = fmaf(P[entry(z)], part(u, entry(z)), o);
          if (MODE == kDecay) o *= a.q_scale;
          if (MODE == kSsd) o += skip * vt;
          if (has) *op = o;
          op += o_step;
        }
        // The block's decay meets the first token's part in one rounding, as eight tokens' decays would.  A state that only decays takes
        // it with what its own rounding left, which would otherwise be the same in every block and add up (heads of 128 x 128, 500
        // tokens of one decay and sign: 2.6e-7 off against 64 bits without, 0.7e-7 token by token).
        // (The corrected form with a decay per channel, short of registers, decays first: 2.8e-7, 3.0e-7 token by token.)
        constexpr bool REST = MODE == kDecay, FIRST = MODE == kDelta && CHAN;
        f2 ge[CH / 2], gl[CH / 2];
        if (CHAN) {
          ldv2<CH>(ge, B + SM::kGend + lane * CH);
          if (FIRST) {
#pragma unroll
            for (int c = 0; c < CW; ++c)
#pragma unroll
              for (int r = 0; r < CH / 2; ++r) s[c][r] = mul2(s[c][r], ge[r]);
          }
          if (REST) ldv2<CH>(gl, B + SM::kGrest + lane * CH);
        } else {
#pragma unroll
          for (int r = 0; r < CH / 2; ++r) {
            ge[r] = pack2(G[3 * kBT - 1], G[3 * kBT - 1]);
            if (REST) gl[r] = pack2(G[0], G[0]);
          }
        }
        const float* kd = B + (CHAN ? 2 * SM::kRows : 0) + lane * CH;       // keys as they enter the state
#pragma unroll
        for (int t = 0; t < kBT; ++t) {
          f2 y[CH / 2];
          if constexpr (KEEP) {
#pragma unroll
            for (int r = 0; r < CH / 2; ++r) y[r] = kept[t][r];
          } else {
            ldv2<CH>(y, kd + t * DK);
          }
          float uu[CW];
          ldv<CW>(uu, us + t * 4);
          f2 u[CW];
#pragma unroll
          for (int c = 0; c < CW; ++c) u[c] = pack2(uu[c], uu[c]);
#pragma unroll
          for (int r = 0; r < CH / 2; ++r)
#pragma unroll
            for (int c = 0; c < CW; ++c) {
              if (t == 0 && !FIRST) s[c][r] = fma2(s[c][r], ge[r], REST ? fma2(y[r], u[c], mul2(s[c][r], gl[r])) : mul2(y[r], u[c]));
              else s[c][r] = fma2(y[r], u[c], s[c][r]);
            }
        }
        __syncwarp();
        if (lane == 0) {
          // The place is overwritten by another block's bulk copy, so what was read here is released at cluster scope, as far as shared memory
          // goes.  A release of everything takes 900 cycles more, in the walk or in a thread beside it: 4096 tokens of the delta rule
          // 451 us so, 685 by a full release here, 597 by one for two blocks, 728 by one in the preparing warps.
          if (nc > 1)
            asm volatile("fence.release.sync_restrict::shared::cta.cluster;\n\t"
                         "mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(mapa_shared(smem_u32(&done[g % kRing]), g & (nc - 1))) : "memory");
          else
            mbar_arrive(&done[g % kRing]);
        }
      }
#pragma unroll
      for (int r = 0; r < CH; r += 2) {
        float x[2][CW];
#pragma unroll
        for (int c = 0; c < CW; ++c) unpack2(s[c][r / 2], x[0][c], x[1][c]);
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          const int i = lane * CH + r + z;
          if (i >= dim) continue;
          float* dst = sp + static_cast<size_t>(i) * vdim;
          if (wide_s && colw < vdim) {
            stv<CW>(dst, x[z]);
          } else {
#pragma unroll
            for (int c = 0; c < CW; ++c)
              if (colw + c < vdim) dst[c] = x[z][c];
          }
        }
      }
    }
    blocks += nblk;
  }
  if (nc > 1) {                                                        // nothing is on its way to, or read from, a block that is gone
    __syncwarp();
    cluster_arrive();
    cluster_wait();
  }
  pdl_wait();          // the short sequences' kernel, of which nothing is read here, ends before this one does
}

// Portions of up to kShort tokens, token by token.  grid = (column blocks, heads, sequences); 128 threads = 32 rows x 4 columns of
// 4.  16 columns per block, so that a single sequence of 16 heads of 128 still makes 128 blocks, and small blocks, of which an
// SM holds many.  Single tokens are bound by the state's way in and out, which are whole 64-byte rows here, more tokens by
// instructions and, for the delta rule, a barrier per token; their rows are staged and normed together, CT tokens at a time.
// Device time of the call, 16 heads of 128 x 128, delta rule, here and in one kernel of eight lanes per column: 32 sequences of one
// token (67 MB, 10 us at the copy rate) 16 and 30.5 us, of two 20 and 35, of eight 37 and 63.
template <int DK, int MODE, bool CHAN>
__global__ void __launch_bounds__(128)
scan_short_kernel(const ScanArgs a) {
  constexpr int NR = DK / 32, CT = DK * (CHAN ? 2 : 1) <= 128 ? 16 : 8;
  __shared__ __align__(16) float ks[CT][DK], qs[CT][DK], ds[CHAN ? CT : 1][CHAN ? DK : 4], vs[CT][kOneCols];
  __shared__ __align__(16) float red[2][4][kOneCols], sums[CT][4][kOneCols];
  __shared__ float sc[CT][3];                          // decay, write strength, what the read-out is multiplied by
  const int h = blockIdx.y, b = blockIdx.z, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, col0 = blockIdx.x * kOneCols;
  pdl_trigger();
  const int t0 = a.cu_seqlens_q[b], n = static_cast<int>(a.cu_seqlens_q[b + 1]) - t0;
  if (n < 1 || n > kShort) return;
  const bool fresh = static_cast<int>(a.context_lens[b]) == n;
  const int dim = a.dim, vdim = a.vdim, hk = MODE == kDecay ? h : h / (a.heads / a.kv_heads);
  const int c = (tid & 3) * 4, col = col0 + c, row = tid >> 2;
  float* sp = a.state + ((static_cast<size_t>(a.state_slots[b]) * a.heads + h) * dim) * vdim + col;
  const bool wide_s = vdim % 4 == 0 && (reinterpret_cast<uintptr_t>(a.state) & 15) == 0;
  float s[NR][4];
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const int i = row + r * 32;
    s[r][0] = s[r][1] = s[r][2] = s[r][3] = 0.f;
    if (!fresh && i < dim && col < vdim) {
      const float* src = sp + static_cast<size_t>(i) * vdim;
      if (wide_s) {
        const float4 v = *reinterpret_cast<const float4*>(src);
        s[r][0] = v.x; s[r][1] = v.y; s[r][2] = v.z; s[r][3] = v.w;
      } else {
#pragma unroll
        for (int x = 0; x < 4; ++x)
          if (col + x < vdim) s[r][x] = src[x];
      }
    }
  }
  const bool wide = dim % 4 == 0 && (a.ld_q | a.ld_k) % 4 == 0 && (!CHAN || a.ld_decay % 4 == 0) &&
                    ((reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.k) |
                      (CHAN ? reinterpret_cast<uintptr_t>(a.chan_decay) : 0)) & 15) == 0;
  const float skip = MODE == kSsd && a.d_skip ? a.d_skip[h] : 0.f;
  // sums over the rows: four columns' of a thread over the lanes of these columns (halving the values), then over the warps
  auto meet = [&](const float (&x)[4], float (*to)[kOneCols]) {
    const bool up = lane & 16, up8 = lane & 8;
    float a0 = up ? x[2] : x[0], a1 = up ? x[3] : x[1];
    a0 += __shfl_xor_sync(0xffffffffu, up ? x[0] : x[2], 16);
    a1 += __shfl_xor_sync(0xffffffffu, up ? x[1] : x[3], 16);
    float y = up8 ? a1 : a0;
    y += __shfl_xor_sync(0xffffffffu, up8 ? a0 : a1, 8);
    y += __shfl_xor_sync(0xffffffffu, y, 4);
    if (!(lane & 4)) to[warp][c + (up ? 2 : 0) + (up8 ? 1 : 0)] = y;
  };
  for (int c0 = 0; c0 < n; c0 += CT) {
    const int m = min(CT, n - c0);
    if (c0 > 0) __syncthreads();                       // the tokens before are stored
    constexpr int TPR = DK / 4, RPS = 128 / TPR;       // threads per row, rows at a time
    const int x = tid % TPR * 4;
    for (int r = tid / TPR; r < m; r += RPS) {
      const size_t t = t0 + c0 + r;
      const float* kg = a.k + t * a.ld_k + hk * dim + x;
      const float* qg = a.q + t * a.ld_q + hk * dim + x;
      const float* ag = CHAN ? a.chan_decay + t * a.ld_decay + h * dim + x : nullptr;
      if (wide && x < dim) {
        cp_async16(&ks[r][x], kg);
        cp_async16(&qs[r][x], qg);
        if (CHAN) cp_async16(&ds[CHAN ? r : 0][CHAN ? x : 0], ag);
      } else {
#pragma unroll
        for (int z = 0; z < 4; ++z) {
          const bool in = x + z < dim;                 // the padding past `dim`: no key, no query, decay one
          ks[r][x + z] = in ? kg[z] : 0.f;
          qs[r][x + z] = in ? qg[z] : 0.f;
          if (CHAN) ds[CHAN ? r : 0][CHAN ? x + z : 0] = in ? ag[z] : 1.f;
        }
      }
    }
    cp_async_commit();
    for (int e = tid; e < m * kOneCols; e += 128) {
      const int r = e / kOneCols, cc = e % kOneCols;
      float v = col0 + cc < vdim ? a.v[static_cast<size_t>(t0 + c0 + r) * a.ld_v + h * vdim + col0 + cc] : 0.f;
      vs[r][cc] = MODE == kDecay && a.act ? silu_exact(v) : v;
    }
    if (tid < m) {
      const size_t o = static_cast<size_t>(t0 + c0 + tid) * a.ld_s + h;
      float g = 1.f, w = a.k_scale;
      if (MODE == kDelta) {
        w = sigmoid_f(a.strength[o]);
        if (!CHAN) g = expf(-expf(a.a_log[h]) * softplus_f(a.decay_raw[o] + a.dt_bias[h]));
      } else if (MODE == kSsd) {
        w = softplus_f(a.decay_raw[o] + a.dt_bias[h]);
        g = expf(-expf(a.a_log[h]) * w);
      } else if (!CHAN) {
        g = a.head_decay[h];
      }
      sc[tid][0] = g;
      sc[tid][1] = w;
      if (MODE != kDelta) sc[tid][2] = MODE == kDecay ? a.q_scale : 1.f;
    }
    cp_async_wait<0>();
    __syncthreads();
    if (MODE == kDelta) {                              // a warp per token: unit keys; the query's norm goes to the read-out
      for (int r = warp; r < m; r += 4) {
        float kx[NR], sk = 0.f, sq = 0.f;
#pragma unroll
        for (int i = 0; i < NR; ++i) {
          kx[i] = ks[r][lane + i * 32];
          const float qx = qs[r][lane + i * 32];
          sk += kx[i] * kx[i];
          sq += qx * qx;
        }
        sk = lanes_sum(sk);
        sq = lanes_sum(sq);
        const float ik = 1.f / sqrtf(sk + 1e-6f);
#pragma unroll
        for (int i = 0; i < NR; ++i) ks[r][lane + i * 32] = kx[i] * ik;
        if (lane == 0) sc[r][2] = rsqrtf(static_cast<float>(dim)) / sqrtf(sq + 1e-6f);
      }
      __syncthreads();
    } else if (MODE == kDecay && a.act) {
      for (int e = tid; e < m * DK; e += 128) {
        if (e % DK >= dim) continue;
        ks[e / DK][e % DK] = silu_exact(ks[e / DK][e % DK]);
        qs[e / DK][e % DK] = silu_exact(qs[e / DK][e % DK]);
      }
      __syncthreads();
    }
    for (int t = 0; t < m; ++t) {
      const float g = sc[t][0], w = sc[t][1];
      const float4 vv = *reinterpret_cast<const float4*>(&vs[t][c]);
      const float v[4] = {vv.x, vv.y, vv.z, vv.w};
      float kv[NR], u[4], o[4] = {};
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        kv[r] = ks[t][row + r * 32];
        const float d = CHAN ? ds[CHAN ? t : 0][CHAN ? row + r * 32 : 0] : g;
#pragma unroll
        for (int z = 0; z < 4; ++z) s[r][z] *= d;
      }
      if (MODE == kDelta) {
        float d[4] = {};
#pragma unroll
        for (int r = 0; r < NR; ++r)
#pragma unroll
          for (int z = 0; z < 4; ++z) d[z] += kv[r] * s[r][z];
        meet(d, red[t & 1]);
        __syncthreads();
        float4 y[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) y[i] = *reinterpret_cast<const float4*>(&red[t & 1][i][c]);
        u[0] = w * (v[0] - ((y[0].x + y[1].x) + (y[2].x + y[3].x)));
        u[1] = w * (v[1] - ((y[0].y + y[1].y) + (y[2].y + y[3].y)));
        u[2] = w * (v[2] - ((y[0].z + y[1].z) + (y[2].z + y[3].z)));
        u[3] = w * (v[3] - ((y[0].w + y[1].w) + (y[2].w + y[3].w)));
      } else {
#pragma unroll
        for (int z = 0; z < 4; ++z) u[z] = v[z] * w;
      }
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const float qv = qs[t][row + r * 32];
#pragma unroll
        for (int z = 0; z < 4; ++z) {
          s[r][z] += kv[r] * u[z];
          o[z] += qv * s[r][z];
        }
      }
      meet(o, sums[t]);
    }
    __syncthreads();
    for (int e = tid; e < m * kOneCols; e += 128) {
      const int r = e / kOneCols, cc = e % kOneCols;
      if (col0 + cc < vdim)
        a.out[(static_cast<size_t>(t0 + c0 + r) * a.heads + h) * vdim + col0 + cc] =
            ((sums[r][0][cc] + sums[r][1][cc]) + (sums[r][2][cc] + sums[r][3][cc])) * sc[r][2] + skip * vs[r][cc];
    }
  }
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const int i = row + r * 32;
    if (i < dim && col < vdim) {
      float* dst = sp + static_cast<size_t>(i) * vdim;
      if (wide_s) {
        *reinterpret_cast<float4*>(dst) = make_float4(s[r][0], s[r][1], s[r][2], s[r][3]);
      } else {
#pragma unroll
        for (int x = 0; x < 4; ++x)
          if (col + x < vdim) dst[x] = s[r][x];
      }
    }
  }
}

template <typename... P, typename... A>
static void launch_cluster(void (*kern)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st_, int nc, A... args) {
  cudaLaunchAttribute attr[2]{};
  int na = 0;
  if (pdl_enabled()) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (nc > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = nc;
    attr[na].val.clusterDim.y = attr[na].val.clusterDim.z = 1;
    ++na;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st_;
  cfg.attrs = attr;
  cfg.numAttrs = na;
  cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}
// Tokens of a sequence above which two, and four, neighbouring blocks of a head share what they prepare; shorter ones end before that pays for the
// clusters' start, for a place's way around, and, of four, for the wait until as many SMs are free.  us, one / two / four blocks, heads of 128 x 128 but as
// noted: delta rule, 16 heads, 8 x 64 tokens 65.5 / 68 / 74, 8 x 100 94.4 / 93.1 / 96.2, 64 x 200 1123 / 997 / 1134, 8 x 300 236 / 220 / 216, 1 x 2000 267 /
// 263 / 219; decayed, 16 heads, 8 x 100 67.7 / 67.9 / 73.8, 64 x 200 804 / 714 / 839, 8 x 300 167 / 157 / 158, 1 x 2000 191 / 174 / 166; delta, a decay per
// channel, 256 x 256, 32 x 40 330 / 304 / 350, 1 x 128 48.2 / 49.5 / 44.6.  (The bits are the same.)
template <int DK, int MODE, bool CHAN> struct ScanShare {
  static constexpr int kTwo = MODE != kDelta ? 112 : DK <= 128 ? 64 : 32;
  static constexpr int kFour = MODE != kDelta ? (DK <= 128 ? 512 : 256) : CHAN && DK > 128 ? 112 : 256;
};
// share: 1, 2 or 4 blocks, where there are as many
template <int DK, int MODE, bool CHAN, int WW>
static void launch_scan_ww(const ScanArgs& a, int z, int above, int to, int share, int* err, cudaStream_t st_) {
  using SM = ScanSmem<DK, CHAN, WW>;
  auto kern = scan_kernel<DK, MODE, CHAN, WW>;
  static OncePerDevice sized;
  if (!allow_smem(sized, kern, SM::kBytes)) return;
  const int cols = (a.vdim + SM::kCols - 1) / SM::kCols;
  // a few blocks per SM, each taking every so many sequences; of a launch for long ones only, which may have none, one per SM (32 sequences of 40
  // tokens, 16 heads of 128 x 128: four waves of blocks that only look took 5 of 111 us)
  z = std::max(1, std::min(z, (above > kShort ? 1 : 4) * sm_count() / (cols * a.heads)));
  const int nc = share == 1 || cols % 2 ? 1 : share == 2 || cols % 4 ? 2 : 4;
  launch_cluster(kern, dim3(cols, a.heads, z), WW * 32 + 256, SM::kBytes, st_, nc, a, a.num_seqs, above, to, nc, err);
  B200_CUDA_LAUNCH_CHECK();
}
template <int DK, int MODE, bool CHAN>
static void launch_scan_dk(const ScanArgs& a, int num_tokens, cudaStream_t st_) {
  int* err = wait_error_flag();
  if (!err) {
    set_error(2, "scan: no host-visible memory");
    return;
  }
  // Which kernel walks a sequence is a matter of its own length, so that its bits do not depend on the step's other sequences.  Up to
  // kShort tokens, whatever their number, token by token is as fast or faster.  Delta rule, heads of 128 x 128, token by token and
  // in blocks: 1 sequence of 16 tokens of 16 heads 9.2 and 9.4 us, 2 10.8 and 10.1, 8 22 and 31, 32 of 12 tokens 51 and 78; of 20
  // tokens 1 sequence 11.5 and 10.5, 4 18.6 and 20.8.  In a step with longer sequences its walk stood before theirs.
  auto brief = DK == 64 && a.dim <= 32 ? scan_short_kernel<DK == 64 ? 32 : DK, MODE, CHAN> : scan_short_kernel<DK, MODE, CHAN>;
  // (a plain launch: the walks below start under it and write before they wait for it)
  brief<<<dim3((a.vdim + kOneCols - 1) / kOneCols, a.heads, a.num_seqs), 128, 0, st_>>>(a);
  B200_CUDA_LAUNCH_CHECK();
  // The walk of the longer sequences starts beside it: they share what they read, and nothing that they write (a sequence of 400 tokens and
  // 32 of 4, 16 heads of 128 x 128, a decay per channel: 101.5 so; 105 one after the other).  It writes before it waits for the kernel
  // in front, at its end, which is only right behind a plain launch, or another of its own kind, that has begun after all earlier ones ended.
  auto walk = [&](int above, int to, int share) {
    // sequences that can be that long: none in a step of few tokens, as of decoded ones
    const int most = num_tokens > 0 ? std::min(a.num_seqs, num_tokens / (above + 1)) : a.num_seqs;
    if (most == 0) return;
    // 16 columns per block while that leaves a block per SM at most, 32 beyond: one sequence of 4096 tokens of 16 heads of
    // 128 x 128 (128 or 64 blocks) 634 and 883 us, four of 1000 (512 or 256 blocks) 655 and 539 us
    const bool narrow = (a.vdim + 15) / 16 * a.heads * (above > kShort ? most : a.num_seqs) <= sm_count();
    if (narrow) launch_scan_ww<DK, MODE, CHAN, 4>(a, most, above, to, share, err, st_);
    else launch_scan_ww<DK, MODE, CHAN, 8>(a, most, above, to, share, err, st_);
  };
  using Share = ScanShare<DK, MODE, CHAN>;
  constexpr int kAny = 1 << 30;
  const int mean = num_tokens > 0 ? num_tokens / a.num_seqs : kAny;
  if (mean > Share::kTwo) {
    walk(kShort, kAny, mean > Share::kFour ? 4 : 2);
  } else if (num_tokens <= std::max(256, 4 * Share::kTwo)) {
    walk(kShort, kAny, 1);
  } else {
    // Short sequences on average, among them perhaps the long portion of a prompt beside decoded tokens: each in the launch for its length.
    // A prompt of 2000 tokens and 32 single ones, all in the form for short ones and so, us: delta rule, 16 heads of 128 x 128 372 and 344, decayed 288 and 257.
    walk(Share::kTwo, kAny, 4);
    walk(kShort, Share::kTwo, 1);
  }
}
// dim: rows of the state; at most 256 (the caller has checked)
template <int MODE, bool CHAN>
static void launch_scan(const ScanArgs& a, int num_tokens, cudaStream_t st_) {
  if (a.dim <= 64) launch_scan_dk<64, MODE, CHAN>(a, num_tokens, st_);
  else if (a.dim <= 128) launch_scan_dk<128, MODE, CHAN>(a, num_tokens, st_);
  else launch_scan_dk<256, MODE, CHAN>(a, num_tokens, st_);
}

// out[t, c] = sigmoid(z)^(1 / tau) with z = bias[c] + sum_r w2[c, r] * low[t, r]: the per-channel decay of gated linear
// attention from the low-rank half of its projection.  Computed as exp(log sigmoid(z) / tau), all fp32.
// a_log != NULL (kind 1): out[t, c] = exp(-exp(a_log[c / a_period]) * softplus(z)), the decay of a gated delta rule per
// head and key channel.
// grid = (channel blocks, token tiles): a thread owns one channel and kDecayTile tokens; the tokens' low-rank rows sit in
// shared memory, entry by entry (four tokens per load), the channel's row of w2 is read once per tile (each thread whole sectors),
// the stores are coalesced.  3001 tokens of 1024 channels, rank 16: 24 us with one token per load, 17 with four.
constexpr int kDecayTile = 16;
__global__ void __launch_bounds__(256)
lowrank_decay_kernel(float* __restrict__ out, const float* __restrict__ low, int ld_low, const float* __restrict__ w2,
                     const float* __restrict__ bias, float inv_tau, const float* __restrict__ a_log, int a_period, int T,
                     int C, int rank) {
  extern __shared__ __align__(16) float lr[];          // [rank][kDecayTile]
  const int t0 = blockIdx.y * kDecayTile, nt = min(kDecayTile, T - t0);
  for (int e = threadIdx.x; e < kDecayTile * rank; e += blockDim.x) {
    const int t = e % kDecayTile;
    lr[e] = t < nt ? low[static_cast<size_t>(t0 + t) * ld_low + e / kDecayTile] : 0.f;
  }
  __syncthreads();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  float z[kDecayTile];
  const float b = bias ? bias[c] : 0.f;
#pragma unroll
  for (int i = 0; i < kDecayTile; ++i) z[i] = b;
  const float* w = w2 + static_cast<size_t>(c) * rank;
  auto add = [&](float wv, int r) {
#pragma unroll
    for (int i = 0; i < kDecayTile; i += 4) {
      const float4 l = *reinterpret_cast<const float4*>(lr + r * kDecayTile + i);
      z[i] += wv * l.x; z[i + 1] += wv * l.y; z[i + 2] += wv * l.z; z[i + 3] += wv * l.w;
    }
  };
  int r = 0;
  if (rank % 4 == 0 && (reinterpret_cast<uintptr_t>(w2) & 15) == 0) {
    for (; r < rank; r += 4) {
      const float4 v = *reinterpret_cast<const float4*>(w + r);
      add(v.x, r); add(v.y, r + 1); add(v.z, r + 2); add(v.w, r + 3);
    }
  }
  for (; r < rank; ++r) add(w[r], r);
#pragma unroll
  for (int i = 0; i < kDecayTile; ++i) {
    if (i >= nt) break;
    if (a_log) {
      out[static_cast<size_t>(t0 + i) * C + c] = expf(-expf(a_log[c / a_period]) * softplus_f(z[i]));
      continue;
    }
    const float ls = z[i] >= 0.f ? -log1pf(expf(-z[i])) : z[i] - log1pf(expf(z[i]));
    out[static_cast<size_t>(t0 + i) * C + c] = expf(ls * inv_tau);
  }
}

void launch_short_conv_silu(float* out, int ldo, const float* x, int ldx, const float* taps_w, const float* bias,
                            float* state, const int32_t* slots, const uint32_t* cu, const uint32_t* ctx, int num_seqs,
                            int num_rows, int C, int taps, cudaStream_t st_) {
  if (num_seqs <= 0 || C <= 0 || num_rows <= 0) return;
  if (taps < 1 || taps > kMaxTaps) {
    set_error(1, "short_conv: between 1 and 8 taps are supported");
    return;
  }
  if (out == x) {
    set_error(1, "short_conv: the output must not alias the input (chunks of a sequence run in parallel)");
    return;
  }
  const dim3 grid((C + 127) / 128, num_seqs, (num_rows + kConvChunk - 1) / kConvChunk);
  const dim3 sgrid((C + 127) / 128, num_seqs);
#define B200_CONV(K)                                                                                              \
  case K:                                                                                                         \
    short_conv_silu_kernel<K><<<grid, 128, 0, st_>>>(out, ldo, x, ldx, taps_w, bias, state, slots, cu, ctx, C); \
    if (K > 1) short_conv_state_kernel<K><<<sgrid, 128, 0, st_>>>(x, ldx, state, slots, cu, ctx, C);           \
    break
  switch (taps) {
    B200_CONV(1); B200_CONV(2); B200_CONV(3); B200_CONV(4); B200_CONV(5); B200_CONV(6); B200_CONV(7); B200_CONV(8);
  }
#undef B200_CONV
  B200_CUDA_LAUNCH_CHECK();
}

void launch_delta_rule(float* out, const float* q, const float* k, const float* v, int ld, const float* b_raw,
                       const float* a_raw, int ld_ba, const float* a_log, const float* dt_bias, const float* chan_decay,
                       int ld_decay, float* state, const int32_t* slots, const uint32_t* cu, const uint32_t* ctx,
                       int num_seqs, int heads, int kv_heads, int dim, int vdim, cudaStream_t st_, int num_tokens) {
  if (num_seqs <= 0) return;
  if (dim > 256) {
    set_error(1, "delta_rule: key dimension above 256 is not supported");
    return;
  }
  const ScanArgs s{out, q, k, v, b_raw, a_raw, a_log, dt_bias, nullptr, nullptr, chan_decay, state, slots, cu, ctx, num_seqs,
                   ld, ld, ld, ld_ba, ld_decay, heads, kv_heads, dim, vdim, 0, 1.f, 1.f};
  if (chan_decay) launch_scan<kDelta, true>(s, num_tokens, st_);
  else launch_scan<kDelta, false>(s, num_tokens, st_);
}

void launch_ssd_scan(float* out, const float* x, const float* Bm, const float* Cm, int ld, const float* dt_raw,
                     int ld_dt, const float* a_log, const float* dt_bias, const float* d_skip, float* state,
                     const int32_t* slots, const uint32_t* cu, const uint32_t* ctx, int num_seqs, int heads, int groups,
                     int nstate, int vdim, cudaStream_t st_, int num_tokens) {
  if (num_seqs <= 0) return;
  if (nstate > 256) {
    set_error(1, "ssd_scan: state size above 256 is not supported");
    return;
  }
  const ScanArgs s{out, Cm, Bm, x, nullptr, dt_raw, a_log, dt_bias, d_skip, nullptr, nullptr, state, slots, cu, ctx, num_seqs,
                   ld, ld, ld, ld_dt, 0, heads, groups, nstate, vdim, 0, 1.f, 1.f};
  launch_scan<kSsd, false>(s, num_tokens, st_);
}

void launch_lowrank_decay(float* out, const float* low, int ld_low, const float* w2, const float* bias, float tau,
                          const float* a_log, int a_period, int T, int C, int rank, cudaStream_t st_) {
  if (T <= 0 || C <= 0) return;
  if (rank <= 0 || rank > 512) {
    set_error(1, "lowrank_decay: the rank must be between 1 and 512");
    return;
  }
  const dim3 grid((C + 255) / 256, (T + kDecayTile - 1) / kDecayTile);
  lowrank_decay_kernel<<<grid, 256, static_cast<size_t>(kDecayTile) * rank * 4, st_>>>(
      out, low, ld_low, w2, bias, a_log ? 0.f : 1.f / tau, a_log, a_period > 0 ? a_period : 1, T, C, rank);
  B200_CUDA_LAUNCH_CHECK();
}

void launch_decay_attn(float* out, const float* q, const float* k, const float* v, int ld, const float* head_decay,
                       const float* chan_decay, int ld_decay, float q_scale, float k_scale, int act, float* state,
                       const int32_t* slots, const uint32_t* cu, const uint32_t* ctx, int num_seqs, int heads, int dim,
                       int vdim, cudaStream_t st_, int num_tokens) {
  if (num_seqs <= 0) return;
  if (dim > 256) {
    set_error(1, "decay_attn: key dimension above 256 is not supported");
    return;
  }
  const ScanArgs s{out, q, k, v, nullptr, nullptr, nullptr, nullptr, nullptr, head_decay, chan_decay, state, slots, cu, ctx,
                   num_seqs, ld, ld, ld, 0, ld_decay, heads, heads, dim, vdim, act, q_scale, k_scale};
  if (chan_decay) launch_scan<kDecay, true>(s, num_tokens, st_);
  else launch_scan<kDecay, false>(s, num_tokens, st_);
}

void launch_scan_args(const b200_scan_args& a, int kind, int num_tokens, cudaStream_t st_) {
  if (a.num_seqs <= 0) return;
  if (a.dim > 256) {
    set_error(1, "scan: key dimension (state size) above 256 is not supported");
    return;
  }
  if (kind == kSsd) launch_scan<kSsd, false>(a, num_tokens, st_);
  else if (kind == kDelta && a.chan_decay) launch_scan<kDelta, true>(a, num_tokens, st_);
  else if (kind == kDelta) launch_scan<kDelta, false>(a, num_tokens, st_);
  else if (a.chan_decay) launch_scan<kDecay, true>(a, num_tokens, st_);
  else launch_scan<kDecay, false>(a, num_tokens, st_);
}

}  // namespace b200

extern "C" {
void b200_scan(const b200_scan_args* a, int32_t kind, int64_t stream) { b200_scan_rows(a, kind, 0, stream); }
void b200_scan_rows(const b200_scan_args* a, int32_t kind, int32_t num_tokens, int64_t stream) {
  B200_CHECK_ARG(a && a->out && a->q && a->k && a->v && a->state && a->state_slots && a->cu_seqlens_q && a->context_lens &&
                     a->heads > 0 && a->kv_heads > 0 && a->heads % a->kv_heads == 0 && a->dim > 0 && a->vdim > 0 &&
                     kind >= b200::kDelta && kind <= b200::kSsd &&
                     (kind == b200::kDecay ? (a->head_decay != nullptr) != (a->chan_decay != nullptr) && a->kv_heads == a->heads
                      : kind == b200::kSsd ? a->decay_raw && a->a_log && a->dt_bias
                                           : a->strength && (a->chan_decay || (a->decay_raw && a->a_log && a->dt_bias))),
                 "scan: bad arguments");
  b200::launch_scan_args(*a, kind, num_tokens, reinterpret_cast<cudaStream_t>(stream));
}
void b200_short_conv_silu(float* out, int32_t ldo, const float* x, int32_t ldx, const float* taps_w, const float* bias,
                          float* state, const int32_t* state_slots, const uint32_t* cu_seqlens_q,
                          const uint32_t* context_lens, int32_t num_seqs, int32_t num_tokens, int32_t channels,
                          int32_t taps, int64_t stream) {
  B200_CHECK_ARG(out && x && taps_w && state && state_slots && cu_seqlens_q && context_lens, "short_conv: bad arguments");
  b200::launch_short_conv_silu(out, ldo, x, ldx, taps_w, bias, state, state_slots, cu_seqlens_q, context_lens, num_seqs,
                               num_tokens, channels, taps, reinterpret_cast<cudaStream_t>(stream));
}
void b200_delta_rule(float* out, const float* q, const float* k, const float* v, int32_t ld, const float* b_raw,
                     const float* a_raw, int32_t ld_ba, const float* a_log, const float* dt_bias, float* state,
                     const int32_t* state_slots, const uint32_t* cu_seqlens_q, const uint32_t* context_lens,
                     int32_t num_seqs, int32_t heads, int32_t kv_heads, int32_t dim, int32_t vdim, int64_t stream) {
  B200_CHECK_ARG(out && q && k && v && b_raw && a_raw && a_log && dt_bias && state && state_slots && cu_seqlens_q &&
                     context_lens && heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && dim > 0 && vdim > 0,
                 "delta_rule: bad arguments");
  b200::launch_delta_rule(out, q, k, v, ld, b_raw, a_raw, ld_ba, a_log, dt_bias, nullptr, 0, state, state_slots,
                          cu_seqlens_q, context_lens, num_seqs, heads, kv_heads, dim, vdim,
                          reinterpret_cast<cudaStream_t>(stream));
}
void b200_delta_rule_chan(float* out, const float* q, const float* k, const float* v, int32_t ld, const float* b_raw,
                          int32_t ld_b, const float* chan_decay, int32_t ld_decay, float* state,
                          const int32_t* state_slots, const uint32_t* cu_seqlens_q, const uint32_t* context_lens,
                          int32_t num_seqs, int32_t heads, int32_t kv_heads, int32_t dim, int32_t vdim, int64_t stream) {
  B200_CHECK_ARG(out && q && k && v && b_raw && chan_decay && state && state_slots && cu_seqlens_q && context_lens &&
                     heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && dim > 0 && vdim > 0,
                 "delta_rule_chan: bad arguments");
  b200::launch_delta_rule(out, q, k, v, ld, b_raw, nullptr, ld_b, nullptr, nullptr, chan_decay, ld_decay, state,
                          state_slots, cu_seqlens_q, context_lens, num_seqs, heads, kv_heads, dim, vdim,
                          reinterpret_cast<cudaStream_t>(stream));
}
void b200_ssd_scan(float* out, const float* x, const float* Bm, const float* Cm, int32_t ld, const float* dt_raw,
                   int32_t ld_dt, const float* a_log, const float* dt_bias, const float* d_skip, float* state,
                   const int32_t* state_slots, const uint32_t* cu_seqlens_q, const uint32_t* context_lens,
                   int32_t num_seqs, int32_t heads, int32_t groups, int32_t nstate, int32_t vdim, int64_t stream) {
  B200_CHECK_ARG(out && x && Bm && Cm && dt_raw && a_log && dt_bias && state && state_slots && cu_seqlens_q &&
                     context_lens && heads > 0 && groups > 0 && heads % groups == 0 && nstate > 0 && vdim > 0,
                 "ssd_scan: bad arguments");
  b200::launch_ssd_scan(out, x, Bm, Cm, ld, dt_raw, ld_dt, a_log, dt_bias, d_skip, state, state_slots, cu_seqlens_q,
                        context_lens, num_seqs, heads, groups, nstate, vdim, reinterpret_cast<cudaStream_t>(stream));
}
void b200_lowrank_decay(float* out, const float* low, int32_t ld_low, const float* w2, const float* bias, float tau,
                         int32_t num_tokens, int32_t channels, int32_t rank, int64_t stream) {
  B200_CHECK_ARG(out && low && w2 && tau > 0.f && channels > 0 && rank > 0 && rank <= 512, "lowrank_decay: bad arguments (rank up to 512)");
  b200::launch_lowrank_decay(out, low, ld_low, w2, bias, tau, nullptr, 1, num_tokens, channels, rank,
                             reinterpret_cast<cudaStream_t>(stream));
}
void b200_lowrank_decay_ex(float* out, const float* low, int32_t ld_low, const float* w2, const float* bias, float tau,
                           int32_t kind, const float* a_log, int32_t a_period, int32_t num_tokens, int32_t channels,
                           int32_t rank, int64_t stream) {
  B200_CHECK_ARG(out && low && w2 && channels > 0 && rank > 0 && rank <= 512 &&
                     (kind == 0 ? tau > 0.f : (kind == 1 && a_log && a_period > 0 && channels % a_period == 0)),
                 "lowrank_decay: bad arguments (rank up to 512; kind 0 needs tau, kind 1 a_log)");
  b200::launch_lowrank_decay(out, low, ld_low, w2, bias, tau, kind == 1 ? a_log : nullptr, a_period, num_tokens, channels,
                             rank, reinterpret_cast<cudaStream_t>(stream));
}
void b200_decay_attn(float* out, const float* q, const float* k, const float* v, int32_t ld, const float* head_decay,
                     const float* chan_decay, int32_t ld_decay, float q_scale, float k_scale, int32_t act, float* state,
                     const int32_t* state_slots, const uint32_t* cu_seqlens_q, const uint32_t* context_lens,
                     int32_t num_seqs, int32_t heads, int32_t dim, int32_t vdim, int64_t stream) {
  B200_CHECK_ARG(out && q && k && v && ((head_decay != nullptr) != (chan_decay != nullptr)) && state && state_slots &&
                     cu_seqlens_q && context_lens && heads > 0 && dim > 0 && vdim > 0,
                 "decay_attn: bad arguments (exactly one of head_decay / chan_decay)");
  b200::launch_decay_attn(out, q, k, v, ld, head_decay, chan_decay, ld_decay, q_scale, k_scale, act, state, state_slots,
                          cu_seqlens_q, context_lens, num_seqs, heads, dim, vdim, reinterpret_cast<cudaStream_t>(stream));
}
}
