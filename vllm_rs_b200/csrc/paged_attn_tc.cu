// Softmax attention over paged bf16 caches on tcgen05 tensor cores, for the hybrid decoders: windowed grouped-head
// attention (window_attn.cu has the list of options) and latent attention (one shared row per token whose first vdim
// entries are the values).  Queries, scores, softmax and sums are fp32; the operands of both products are bf16.
//
// A block owns 128 rows = (128 / group) tokens x the `group` query heads of ONE key head (latent attention: all heads),
// so that every key page is fetched once for all of them, and walks the pages (64 tokens) that its rows see: first those
// that hold kept tokens outside the window, then the window.
//   S  = Q K^T    fp32 [128 x 64] in TMEM.  Q was rounded to bf16 once: in shared memory (SW128, K-major) or, where the key
//                 rows are so long that Q and the page ring do not fit together, its first q_tm blocks of 64 in TMEM
//   P  = softmax  two threads per row, half of a page's keys each: options and mask on the fp32 scores, running maximum (the accumulator is rescaled whenever a
//                 row's maximum grows: letting it lag by up to 2^8 saves 3 - 10 % of the time, but the largest weight of a
//                 row then is not 1 and is rounded like the others, 4 - 8 % more error against 64 bits), bf16 P to TMEM.
//                 Steps of few rows take every page's own maximum: its largest weight is exact then, as the largest of every
//                 split was where a row's keys were split over 16 blocks (32 tokens over 2048 keys, 32 heads over 8: error
//                 0.00280 with the running maximum, 0.00276 with 16 splits, 0.00268 here; 59 -> 62 us)
//   O += P V      fp32 [128 x up to 256] in TMEM; V = page as an MN-major operand
// Warp 0 fetches pages by block-table index (TMA, K ring | V ring), warp 1 issues the MMAs (S of page j + 1 before P V of
// page j), warps 2-9 own the rows: two warps share 32 of them, exchange their halves' maxima in shared memory at a barrier of the
// two, and rescale and write half of the columns each.  (One thread per row has a page's 64 scores in one chain of waits: 98 / 62 / 680
// us for the three cases below, in turn with others, where two took 90 / 58 / 577.  More warps also stage the queries faster.)  Latent rows (kv_rank 512: O would need all 512 TMEM columns) are walked in passes of up to
// 256 value columns; the scores are computed again in every pass (1.5x the products, still far from the 8 mma.sync
// warps' rate that made 128-row tiles of 16 rows x 1 head re-read every page 64 times).  In a pass the page blocks that are
// also values stay until P V has read them (V ring), the rest is released after S (K ring).
//
// Bound: tensor cores for prompts (per page 2 * 128 * 64 * (dim * passes + vdim) flop against 64 * dim * 2 bytes from L2),
// HBM for steps of few rows, whose keys are split over blocks; window_attn_merge / latent_attn_merge then finish.
// Measured, whole calls in turn with others, mma.sync kernels -> here: window 1024, 4096 rows, 16 heads of 128 over 4: 622 -> 88 us
// (340 TFLOP/s; what bounds it is the softmax warps, then the start and the drain of 128 blocks); latent, 2 x 2048 rows, 32 heads, rank 512:
// 7766 -> 561 us (533 TFLOP/s useful, 810 issued); 32 tokens over 2048 keys, 32 heads over 8: 317 -> 57.6 us (35 at HBM rate): 256 blocks
// of 33 pages in turn, with four rows in one pair of the row warps.
#include "paged_attn_tc.cuh"
#include "f32x2.cuh"

#include <algorithm>

namespace b200 {
using namespace seqmix;
namespace hat {

constexpr int kRows = 128, kTok = 64, kRowWarps = 8, kThreads = 64 + kRowWarps * 32;
constexpr int kHalf = kTok / 2;           // keys of a page (and half of a pass's columns) that one of a row's two threads has
constexpr int kBlk = kTok * 128;          // a page's 64 x 64 block: 64 swizzled rows of 128 bytes
constexpr int kTailBlk = kTok * 64;       // the last 32 columns: 64 rows of 64 bytes
constexpr int kQBlk = kRows * 128, kQTail = kRows * 64;
constexpr int kMaxStages = 4;
constexpr float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f;
constexpr float kNone = -1e30f;           // a reference maximum before any key was seen
constexpr float kPageLag = 8.f;           // how far below the largest score the reference may fall: sums stay 2^8 within range

struct Args {
  AttnTcProblem p;
  int group, tq;                          // query heads per key head; tokens per block
  int kblk, tail, vblk, passes, ppc;      // 64-wide blocks of a key row (+ 32-wide tail), of a value row; passes; passes per block
  int shared, q_tm, sk, sv;               // values inside the key rows; query blocks in TMEM; ring stages
  int k_stage, v_stage, q_bytes, tmem_cols, page_ref;
  int wide_q, wide_out;                   // on 32 bytes
  uint32_t by_group;                      // row / group = row * by_group >> 16 (row < 256)
  int* err;
};

// Operand descriptors, upper words (version 1, SBO; layout 2 = SW128, 4 = SW64).  The lower word is the address in 16-byte
// units under the LBO: unused for K-major rows (1); 8 KB between the 64-column chunks of the MN-major values.
constexpr uint32_t kHiSw128 = (1024 >> 4) | (1u << 14) | (2u << 29), kHiSw64 = (512 >> 4) | (1u << 14) | (4u << 29);
__device__ __forceinline__ uint32_t desc_k(uint32_t saddr) { return (saddr >> 4) | (1u << 16); }
__device__ __forceinline__ uint32_t desc_mn(uint32_t saddr) { return (saddr >> 4) | (uint32_t(kBlk >> 4) << 16); }
// One lane (lead != 0) issues; the warp runs the loop around it together, so that addresses stay uniform.
__device__ __forceinline__ void mma_ss(uint32_t lead, uint32_t d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                       uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 q, %0, 0;\n\tsetp.ne.b32 p, %7, 0;\n\t"
      "mov.b64 da, {%2, %3};\n\tmov.b64 db, {%4, %5};\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%1], da, db, %6, p;\n\t}\n" ::"r"(lead),
      "r"(d), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void mma_ts(uint32_t lead, uint32_t d, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                       uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 db;\n\t"
      "setp.ne.b32 q, %0, 0;\n\tsetp.ne.b32 p, %6, 0;\n\t"
      "mov.b64 db, {%3, %4};\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%1], [%2], db, %5, p;\n\t}\n" ::"r"(lead),
      "r"(d), "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void commit(uint32_t lead, uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %0, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%1];\n\t}\n" ::"r"(lead),
      "r"(smem_u32(bar))
      : "memory");
}
// 32 bytes of a lane at once: the scattered rows of a warp are a line each to the load and store units
__device__ __forceinline__ void ld32(float4& lo, float4& hi, const float* p, bool wide) {
  if (wide)
    asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(lo.x), "=f"(lo.y), "=f"(lo.z), "=f"(lo.w), "=f"(hi.x), "=f"(hi.y), "=f"(hi.z), "=f"(hi.w) : "l"(p));
  else {
    lo = __ldg(reinterpret_cast<const float4*>(p));
    hi = __ldg(reinterpret_cast<const float4*>(p) + 1);
  }
}
__device__ __forceinline__ void st32(void* p, const uint4& lo, const uint4& hi, bool wide) {
  if (wide)
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(lo.x), "r"(lo.y), "r"(lo.z), "r"(lo.w), "r"(hi.x),
                 "r"(hi.y), "r"(hi.z), "r"(hi.w)
                 : "memory");
  else {
    reinterpret_cast<uint4*>(p)[0] = lo;
    reinterpret_cast<uint4*>(p)[1] = hi;
  }
}
// tanh(y) = y P(y^2) for |y| <= kTanhMax: fit of tanh(y) / y in y^2, relative error 6.6e-8 before rounding
constexpr float kTanhMax = 0.75f;
constexpr float kT0 = 1.f, kT1 = -0.33332958817481995f, kT2 = 0.1332540661096573f, kT3 = -0.05334442853927612f,
                kT4 = 0.019582903012633324f, kT5 = -0.004716253839433193f;
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
      "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
      "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]),
      "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
      : "memory");
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ int first_seen(int pos, int window, int chunk) {
  const int lo = window > 0 ? max(0, pos - window + 1) : 0;
  return chunk > 0 ? max(lo, pos / chunk * chunk) : lo;
}

// Waits do not end the loops around them: once one has given up (*fail), every other returns at once and the loops run out,
// over shared memory and TMEM that stay the block's; what is still in flight then is waited for at the end.
// Ring position: stage and the parity of its current use.
struct Ring {
  int s = 0;
  uint32_t ph = 0;
  __device__ __forceinline__ void next(int stages) {
    if (++s == stages) { s = 0; ph ^= 1; }
  }
};

// CAP: scores are capped; BIAS: a distance bias (slopes or table) joins them.
template <bool CAP, bool BIAS>
__global__ void __launch_bounds__(kThreads, 2)
attn_tc_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap tmap,
               const __grid_constant__ CUtensorMap vmap, const __grid_constant__ Args a) {
  const AttnTcProblem& p = a.p;
  pdl_trigger();       // the merge of split keys may start (launch_attn_merge)
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int G = a.group, kvh = blockIdx.y, vh = kvh % p.v_heads;
  // ---- which tokens: tile (gridDim.x - 1 - blockIdx.x) of the sequences' tiles, so that the latest (longest) go first
  int b = -1, tile = 0;
  {
    const int want = static_cast<int>(gridDim.x - 1 - blockIdx.x);
    int before = 0;
    for (int s0 = 0; s0 < p.num_seqs && b < 0; s0 += 32) {
      const int s = s0 + lane;
      const int n = s < p.num_seqs ? static_cast<int>(p.cu[s + 1] - p.cu[s]) : 0;
      const int mine = (n + a.tq - 1) / a.tq;
      int inc = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
      }
      const bool here = want >= before + inc - mine && want < before + inc;
      const unsigned hit = __ballot_sync(0xffffffffu, here);
      if (hit) {
        const int src = __ffs(hit) - 1;
        b = s0 + src;
        tile = want - before - __shfl_sync(0xffffffffu, inc - mine, src);
      }
      before += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (b < 0) return;
  }
  const int seq0 = static_cast<int>(p.cu[b]), nq = static_cast<int>(p.cu[b + 1]) - seq0;
  const int row0 = seq0 + tile * a.tq;                       // first token row
  const int nt = min(a.tq, nq - tile * a.tq), nrows = nt * G;
  const int p_ctx = static_cast<int>(p.ctx[b]);
  const int pos0 = p_ctx - nq + tile * a.tq, pos_last = pos0 + nt - 1;
  const int key_lo = first_seen(pos0, p.window, p.chunk);
  const int wpage = key_lo / kTok;
  const int nkept = min(wpage, (min(max(p.keep_first, 0), key_lo) + kTok - 1) / kTok);
  const int ntiles = nkept + pos_last / kTok - wpage + 1;
  const int npz = a.passes / a.ppc, sp = blockIdx.z / npz, pass0 = (blockIdx.z % npz) * a.ppc;
  const int per = (ntiles + p.nsplit - 1) / p.nsplit;
  const int j0 = sp * per, n = __shfl_sync(0xffffffffu, min(ntiles, j0 + per) - j0, 0);   // this block's pages
  const int nwarps = (nrows + 31) / 32;                      // row warps that have a row
  const int vcols = a.vblk * 64;                             // value columns of a pass (the last one may have fewer)

  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* q_smem = smem;
  uint8_t* k_smem = q_smem + a.q_bytes;
  uint8_t* v_smem = k_smem + a.sk * a.k_stage;
  float* s_max = reinterpret_cast<float*>(v_smem + a.sv * a.v_stage);       // [page parity][half of the keys][row]
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_max + 4 * kRows);
  uint64_t* k_full = bars;
  uint64_t* k_empty = k_full + kMaxStages;
  uint64_t* v_full = k_empty + kMaxStages;
  uint64_t* v_empty = v_full + kMaxStages;
  uint64_t* q_full = v_empty + kMaxStages;
  uint64_t* s_full = q_full + 1;
  uint64_t* s_free = q_full + 2;
  uint64_t* p_full = q_full + 3;
  uint64_t* pv_done = q_full + 4;
  uint64_t* drained = q_full + 5;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(q_full + 6);
  volatile int* fail = reinterpret_cast<volatile int*>(tmem_ptr + 1);

  if (smem_u32(smem) & 1023) {             // the swizzles' atoms; dynamic shared memory without static one begins on them
    if (threadIdx.x == 0) *reinterpret_cast<volatile int*>(a.err) = 1;
    return;
  }
  if (n <= 0) {                            // a split without keys leaves an empty part
    for (int e = threadIdx.x; e < nrows * a.ppc * vcols; e += kThreads) {
      const int r = e / (a.ppc * vcols), c = pass0 * vcols + e % (a.ppc * vcols);
      const size_t pi = (static_cast<size_t>(row0 + r / G) * p.heads + kvh * G + r % G) * p.nsplit + sp;
      if (c < p.vdim) p.part_o[pi * p.vdim + c] = 0.f;
      if (c == 0) {
        p.part_ml[pi * 2] = kNone;
        p.part_ml[pi * 2 + 1] = 0.f;
      }
    }
    return;
  }

  if (threadIdx.x == 0) {
    for (int s = 0; s < a.sk; ++s) { mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1); }
    for (int s = 0; s < a.sv; ++s) { mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1); }
    mbar_init(q_full, kRowWarps);
    mbar_init(s_full, 1);
    mbar_init(s_free, 2 * nwarps);
    mbar_init(p_full, 2 * nwarps);
    mbar_init(pv_done, 1);
    mbar_init(drained, 1);
    *fail = 0;
    fence_barrier_init();
    prefetch_tmap(&kmap);
    prefetch_tmap(&vmap);
    if (a.tail) prefetch_tmap(&tmap);
  }
  if (warp == 1) {
    tmem_alloc(tmem_ptr, a.tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_ptr, 0);
  const uint32_t o_tm = tmem, s_tm = tmem + vcols, p_tm = s_tm + 64, q_tm = p_tm + 32;
  // blocks of value columns in pass x, and the first of them
  auto v_first = [&](int x) { return x * a.vblk; };
  auto v_count = [&](int x) { return min(a.vblk, p.vdim / 64 - x * a.vblk); };
  auto page_of = [&](int j) { return j < nkept ? j : wpage + j - nkept; };

  if (warp == 0) {
    // ------------------------------------------------------------ pages
    if (a.q_tm) mbar_wait_limited(q_full, 0, fail, a.err);      // the rings lend their space to the staging of Q
    const uint32_t* bt = p.block_tables + static_cast<size_t>(b) * p.max_blocks;
    Ring kr, vr;
    int armed_k = 0, armed_v = 0;           // (a stage that did not come free is not armed again, nor any after it)
    bool free_ = true;
    for (int pi = 0; pi < a.ppc; ++pi) {
      const int vf = v_first(pass0 + pi), vn = v_count(pass0 + pi);
      const int kn = a.shared ? a.kblk - vn : a.kblk;
      for (int base = 0; base < n; base += 32) {
        const int mine = base + lane < n ? static_cast<int>(bt[page_of(j0 + base + lane)]) : 0;
        const int cnt = min(32, n - base);
        for (int jj = 0; jj < cnt; ++jj) {
          const int page = __shfl_sync(0xffffffffu, mine, jj);
          if (elect_one()) {
            free_ = free_ && mbar_wait_limited(&k_empty[kr.s], kr.ph ^ 1, fail, a.err);
            if (free_) {
              uint8_t* kd = k_smem + kr.s * a.k_stage;
              mbar_arrive_expect_tx(&k_full[kr.s], kn * kBlk + a.tail * kTailBlk);
              for (int i = 0; i < kn; ++i) {
                const int blk = a.shared && i >= vf ? i + vn : i;
                tma_load_4d(kd + i * kBlk, &kmap, &k_full[kr.s], blk * 64, kvh, 0, page);
              }
              if (a.tail) tma_load_4d(kd + kn * kBlk, &tmap, &k_full[kr.s], a.kblk * 64, kvh, 0, page);
              ++armed_k;
            }
            free_ = free_ && mbar_wait_limited(&v_empty[vr.s], vr.ph ^ 1, fail, a.err);
            if (free_) {
              uint8_t* vd = v_smem + vr.s * a.v_stage;
              mbar_arrive_expect_tx(&v_full[vr.s], vn * kBlk);
              for (int i = 0; i < vn; ++i)
                tma_load_4d(vd + i * kBlk, &vmap, &v_full[vr.s], (vf + i) * 64, vh, 0, page);
              ++armed_v;
            }
          }
          kr.next(a.sk);
          vr.next(a.sv);
        }
      }
    }
    if (elect_one() && *fail) {             // copies in flight, as the lane that made them counted them, land before the block ends
      for (int s = 0; s < a.sk && s < armed_k; ++s)
        mbar_wait_limited(&k_full[s], ((armed_k - 1 - s) / a.sk) & 1, nullptr, a.err);
      for (int s = 0; s < a.sv && s < armed_v; ++s)
        mbar_wait_limited(&v_full[s], ((armed_v - 1 - s) / a.sv) & 1, nullptr, a.err);
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------ products
    constexpr uint32_t kBf16 = (1u << 7) | (1u << 10);
    constexpr uint32_t idesc_s = make_idesc_f16(kRows, kTok) | kBf16;
    const uint32_t lead = elect_one() ? 1u : 0u;
    const uint32_t q_lo = desc_k(smem_u32(q_smem));
    Ring kr, vr, vr_pv;
    auto wait = [&](uint64_t* bar, uint32_t parity) { mbar_wait_limited(bar, parity, fail, a.err); };
    // S (+)= the queries of block `blk` times a page's block of 64 columns
    auto qk_block = [&](int blk, uint32_t b_lo, uint32_t acc) {
      if (blk < a.q_tm) {
        const uint32_t qa = q_tm + blk * 32;
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) mma_ts(lead, s_tm, qa + ks * 8, b_lo + ks * 2, kHiSw128, idesc_s, ks ? 1u : acc);
      } else {
        const uint32_t a_lo = q_lo + (blk - a.q_tm) * (kQBlk >> 4);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          mma_ss(lead, s_tm, a_lo + ks * 2, kHiSw128, b_lo + ks * 2, kHiSw128, idesc_s, ks ? 1u : acc);
      }
    };
    const uint32_t k_base = desc_k(smem_u32(k_smem)), v_base = desc_k(smem_u32(v_smem)), vm_base = desc_mn(smem_u32(v_smem));
    const uint32_t k_step = a.k_stage >> 4, v_step = a.v_stage >> 4;
    auto issue_qk = [&](int it, int vf, int vn) {
      wait(&k_full[kr.s], kr.ph);
      if (it > 0) wait(s_free, (it - 1) & 1);           // the rows hold S of the page before
      tc_fence_after();
      const uint32_t k_lo = k_base + kr.s * k_step;
      const int kn = a.shared ? a.kblk - vn : a.kblk;
      uint32_t acc = 0;
      for (int i = 0; i < kn; ++i, acc = 1) qk_block(a.shared && i >= vf ? i + vn : i, k_lo + i * (kBlk >> 4), acc);
      if (a.tail) {
        const uint32_t a_lo = q_lo + (a.kblk - a.q_tm) * (kQBlk >> 4), b_lo = k_lo + kn * (kBlk >> 4);
#pragma unroll
        for (int ks = 0; ks < 2; ++ks, acc = 1)
          mma_ss(lead, s_tm, a_lo + ks * 2, kHiSw64, b_lo + ks * 2, kHiSw64, idesc_s, acc);
      }
      commit(lead, &k_empty[kr.s]);
      kr.next(a.sk);
      if (a.shared) {
        wait(&v_full[vr.s], vr.ph);
        tc_fence_after();
        const uint32_t v_lo = v_base + vr.s * v_step;
        for (int i = 0; i < vn; ++i, acc = 1) qk_block(vf + i, v_lo + i * (kBlk >> 4), acc);
        vr.next(a.sv);
      }
      commit(lead, s_full);
    };
    wait(q_full, 0);
    int it = 0;
    issue_qk(0, v_first(pass0), v_count(pass0));
    for (int pi = 0; pi < a.ppc; ++pi) {
      const int vf = v_first(pass0 + pi), vn = v_count(pass0 + pi);
      const uint32_t idesc_o = make_idesc_f16(kRows, vn * 64) | (1u << 16) | kBf16;     // B is MN-major
      for (int j = 0; j < n; ++j, ++it) {
        if (j + 1 < n) issue_qk(it + 1, vf, vn);
        else if (pi + 1 < a.ppc) issue_qk(it + 1, v_first(pass0 + pi + 1), v_count(pass0 + pi + 1));
        wait(p_full, it & 1);
        if (!a.shared) wait(&v_full[vr_pv.s], vr_pv.ph);
        tc_fence_after();
        const uint32_t v_lo = vm_base + vr_pv.s * v_step;
#pragma unroll
        for (int ks = 0; ks < kTok / 16; ++ks)
          mma_ts(lead, o_tm, p_tm + ks * 8, v_lo + ks * (2048 >> 4), kHiSw128, idesc_o, (j > 0 || ks > 0) ? 1u : 0u);
        commit(lead, &v_empty[vr_pv.s]);
        commit(lead, pv_done);
        vr_pv.next(a.sv);
      }
    }
    if (*fail) {                            // products in flight end before TMEM is given back
      commit(lead, drained);
      mbar_wait_limited(drained, 0, nullptr, a.err);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ rows
    // row = TMEM lane; the warps q4 and q4 + 4 share 32 rows: a thread has half of a page's keys and half of the columns
    const int q4 = warp & 3, hf = (warp - 2) >> 2, r = q4 * 32 + lane;
    auto meet = [&] { asm volatile("bar.sync %0, 64;" ::"r"(2 + q4) : "memory"); };
    constexpr int kRowThreads = kRowWarps * 32;
    const int tid = threadIdx.x - 64;
    const uint32_t lane_base = static_cast<uint32_t>(q4 * 32) << 16;
    // ---- stage Q as bf16: coalesced 32-byte reads, chunks of 8 entries (128 rows of 544: 26 000 cycles with divisions and 64-bit
    // addresses per chunk and 16-byte loads, 17 000 without; latent prompt 580 -> 561 us, with the issue
    // behind elect.sync)
    {
      const int cpr = p.dim / 8;
      const int dr = kRowThreads / cpr, dc = kRowThreads % cpr;          // what 256 chunks on are: dr rows and dc chunks
      int row = tid / cpr, c = tid % cpr;
      const float* const first = p.q + (static_cast<size_t>(row0) * p.heads + kvh * G) * p.dim;
      const int skip = p.heads - G;                          // heads between a token's rows and the next one's
      while (row < kRows) {
        constexpr int U = 8;                                 // chunks in flight per thread: 64 KB per block
        float4 lo[U], hi[U];
        const int row_first = row, c_first = c;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          lo[u] = hi[u] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (row < nrows) ld32(lo[u], hi[u], first + ((row + static_cast<int>(row * a.by_group >> 16) * skip) * p.dim + c * 8), a.wide_q);
          row += dr;
          c += dc;
          if (c >= cpr) { c -= cpr; ++row; }
        }
        row = row_first;
        c = c_first;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (row < kRows) {
            uint4 w;
            w.x = pack16x2<true>(lo[u].x, lo[u].y);
            w.y = pack16x2<true>(lo[u].z, lo[u].w);
            w.z = pack16x2<true>(hi[u].x, hi[u].y);
            w.w = pack16x2<true>(hi[u].z, hi[u].w);
            const int blk = c >> 3, c8 = c & 7;
            uint8_t* dst;
            if (blk < a.q_tm) dst = k_smem + blk * kQBlk + row * 128 + ((c8 ^ (row & 7)) << 4);
            else if (blk < a.kblk) dst = q_smem + (blk - a.q_tm) * kQBlk + row * 128 + ((c8 ^ (row & 7)) << 4);
            else dst = q_smem + (a.kblk - a.q_tm) * kQBlk + row * 64 + ((c8 ^ ((row >> 1) & 3)) << 4);
            *reinterpret_cast<uint4*>(dst) = w;
          }
          row += dr;
          c += dc;
          if (c >= cpr) { c -= cpr; ++row; }
        }
      }
      __syncwarp();
      if (a.q_tm) {
        asm volatile("bar.sync 1, %0;" ::"n"(kRowThreads) : "memory");
        for (int blk = hf; blk < a.q_tm; blk += 2) {
          uint32_t w[32];
          const uint8_t* src = k_smem + blk * kQBlk + r * 128;          // (eight lanes' rows lie in different banks)
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint4 v = *reinterpret_cast<const uint4*>(src + ((i ^ (r & 7)) << 4));
            w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
          }
          tmem_st32(q_tm + lane_base + blk * 32, w);
        }
        tc_wait_st();
        tc_fence_before();
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(q_full);
    }
    // ---- this row
    const int tl = min(r / G, nt - 1), h = kvh * G + (r - (r / G) * G);      // rows past nrows repeat the last token's limits
    const bool valid = r < nrows;
    const int pos = pos0 + tl, lo = first_seen(pos, p.window, p.chunk);
    const int lo_last = first_seen(pos_last, p.window, p.chunk);
    const bool with_sink = p.sink && p.nsplit == 1;          // split runs add the sink when the parts are merged
    // what a product becomes a score (or, capped, the argument of tanh) by; scores are in log2 units
    const float sl = CAP ? p.scale / p.softcap : p.scale * kLog2e;
    const float cap2 = p.softcap * kLog2e;
    float slope = 0.f, far_bias = 0.f;
    const float* table = nullptr;
    if (BIAS) {
      slope = (p.slopes && valid) ? p.slopes[h] * kLog2e : 0.f;
      if (p.dist_bias) {
        table = p.dist_bias + static_cast<size_t>(valid ? h : kvh * G) * p.dist_n;
        far_bias = table[p.dist_n - 1] * kLog2e;
      }
    }
    Ring vr;
    int it = 0;
    const int passes = q4 < nwarps ? a.ppc : 0;              // a warp without rows is done
    for (int pi = 0; pi < passes; ++pi) {
      // A sink below every score that counts is no sink (and -inf as a reference makes NaN of a page without a visible key).
      float m_ref = with_sink && valid ? p.sink[h] * kLog2e : kNone, l = with_sink && hf == 0 ? 1.f : 0.f;      // (l: of this half)
      if (m_ref < kNone) {
        m_ref = kNone;
        l = 0.f;
      }
      float m_top = m_ref;                                   // the largest score so far; m_ref where the reference never falls
      const int vn = v_count(pass0 + pi);
      for (int j = 0; j < n; ++j, ++it) {
        const int page0 = page_of(j0 + j) * kTok, base = page0 + hf * kHalf;        // first key of the page, of this half
        mbar_wait_limited(s_full, it & 1, fail, a.err);
        __syncwarp();
        tc_fence_after();
        uint32_t v0[kHalf];
        tmem_ld_x32(s_tm + lane_base + hf * kHalf, v0);
        tc_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(s_free);
        float x[kHalf];
#pragma unroll
        for (int i = 0; i < kHalf; ++i) x[i] = __uint_as_float(v0[i]);
        // x times `mult` is the score; keys outside the mask become -inf
        float mult = sl;
        if (CAP) {
          float big0 = fabsf(x[0]), big1 = fabsf(x[1]);
#pragma unroll
          for (int i = 2; i < kHalf - 2; i += 4) {
            big0 = max3(big0, fabsf(x[i]), fabsf(x[i + 1]));
            big1 = max3(big1, fabsf(x[i + 2]), fabsf(x[i + 3]));
          }
          big0 = max3(big0, fabsf(x[kHalf - 2]), fabsf(x[kHalf - 1]));
          mult = cap2;
          if (__all_sync(0xffffffffu, fmaxf(big0, big1) * sl <= kTanhMax)) {
#pragma unroll
            for (int i = 0; i < kHalf; i += 2) {
              const f2 y = mul2(pack2(x[i], x[i + 1]), pack2(sl, sl)), t = mul2(y, y);
              f2 q = fma2(t, pack2(kT5, kT5), pack2(kT4, kT4));
              q = fma2(t, q, pack2(kT3, kT3));
              q = fma2(t, q, pack2(kT2, kT2));
              q = fma2(t, q, pack2(kT1, kT1));
              q = mul2(y, fma2(t, q, pack2(kT0, kT0)));
              asm("mov.b64 {%0, %1}, %2;" : "=f"(x[i]), "=f"(x[i + 1]) : "l"(q));
            }
          } else {
            // The same products one by one, and tanh(y) = 1 - 2 / (e^(2 y) + 1) past kTanhMax.  Which form a score takes is its
            // own affair: a row's bits do not depend on the rows and heads that share its warp.  (The packed products here too,
            // or a choice per row, made the path above slower: 101 and 107 instead of 99 us for a prompt of 4096, with one thread per row.)
            const float e2 = sl * (2.f * kLog2e);
#pragma unroll
            for (int i = 0; i < kHalf; ++i) {
              const float y = __fmul_rn(x[i], sl), t = __fmul_rn(y, y);
              float q = fmaf(t, kT5, kT4);
              q = fmaf(t, q, kT3);
              q = fmaf(t, q, kT2);
              q = fmaf(t, q, kT1);
              q = __fmul_rn(y, fmaf(t, q, kT0));
              x[i] = fabsf(y) <= kTanhMax ? q : fmaf(-2.f, rcp(ex2(x[i] * e2) + 1.f), 1.f);
            }
          }
        }
        if (BIAS) {
          const float d0 = static_cast<float>(pos - base);
          if (table && pos - (base + kHalf - 1) < p.dist_n - 1) {
#pragma unroll
            for (int i = 0; i < kHalf; ++i)
              x[i] = fmaf(x[i], mult, fmaf(-slope, d0 - i, __ldg(table + max(0, min(pos - base - i, p.dist_n - 1))) * kLog2e));
          } else {
#pragma unroll
            for (int i = 0; i < kHalf; ++i) x[i] = fmaf(x[i], mult, fmaf(-slope, d0 - i, far_bias));
          }
          mult = 1.f;
        }
        if (page0 + kTok - 1 > pos0 || page0 < lo_last) {       // the diagonal, the window's edge, kept tokens
          const int last = pos - base, first = lo - base, kept = p.keep_first - base;
#pragma unroll
          for (int i = 0; i < kHalf; ++i) x[i] = i <= last && (i >= first || i < kept) ? x[i] : -INFINITY;
        }
        float mx0 = max3(x[0], x[1], x[2]), mx1 = max3(x[3], x[4], x[5]);
#pragma unroll
        for (int i = 6; i < kHalf - 2; i += 4) {
          mx0 = max3(mx0, x[i], x[i + 1]);
          mx1 = max3(mx1, x[i + 2], x[i + 3]);
        }
        // of both halves (a place is written again two pages later, behind the barrier of the page between)
        const float own = max3(mx0, mx1, fmaxf(x[kHalf - 2], x[kHalf - 1]));
        float* const top = s_max + (it & 1) * 2 * kRows + r;
        top[hf * kRows] = own;
        meet();
        const float mx = fmaxf(own, top[(hf ^ 1) * kRows]) * mult;
        float corr = 1.f;
        bool grow = false;
        m_top = fmaxf(m_top, mx);
        if (mx > m_ref || (a.page_ref && mx < m_ref && mx > m_top - kPageLag)) {
          corr = ex2(m_ref - mx);
          m_ref = mx;
          grow = true;
        }
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
        uint32_t pk[kHalf / 2];
#pragma unroll
        for (int i = 0; i < kHalf / 2; ++i) {
          const float p0 = ex2(fmaf(x[2 * i], mult, -m_ref)), p1 = ex2(fmaf(x[2 * i + 1], mult, -m_ref));
          pk[i] = pack16x2<true>(p0, p1);
          sum[(2 * i) & 3] += p0;
          sum[(2 * i + 1) & 3] += p1;
        }
        l = fmaf(l, corr, (sum[0] + sum[1]) + (sum[2] + sum[3]));
        // Value rows past the tile's last token may hold anything (later tokens, and what lies behind the sequence), and 0 * NaN
        // is no 0; a single token does not even meet the rows before its window.
        const int v_end = pos_last + 1 - page0, v_lo = nt == 1 && page0 + kTok > p.keep_first ? key_lo - page0 : 0;
        if (v_end < kTok || v_lo > 0) {
          mbar_wait_limited(&v_full[vr.s], vr.ph, fail, a.err);
          uint8_t* vt = v_smem + vr.s * a.v_stage + (r & 7) * 16;
          for (int row = (r >> 3) + hf * nwarps * 4; row < kTok; row += nwarps * 8)
            if (row >= v_end || (row < v_lo && page0 + row >= p.keep_first))
              for (int i = 0; i < vn; ++i) *reinterpret_cast<uint4*>(vt + i * kBlk + row * 128) = make_uint4(0, 0, 0, 0);
          fence_proxy_async();
        }
        vr.next(a.sv);
        if (it > 0) {
          mbar_wait_limited(pv_done, (it - 1) & 1, fail, a.err);           // P and O are the rows' again
          __syncwarp();
          tc_fence_after();
          if (j > 0 && __any_sync(0xffffffffu, grow)) {
#pragma unroll 1
            for (int c0 = hf * vn * 32; c0 < (hf + 1) * vn * 32; c0 += 32) {
              uint32_t o[32];
              tmem_ld_x32(o_tm + lane_base + c0, o);
              tc_wait_ld();
#pragma unroll
              for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
              tmem_st32(o_tm + lane_base + c0, o);
            }
          }
        }
        tmem_st_x16(p_tm + lane_base + hf * (kHalf / 2), pk);
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full);
      }
      mbar_wait_limited(pv_done, (it - 1) & 1, fail, a.err);
      __syncwarp();
      tc_fence_after();
      // ---- the pass's columns of this row
      const size_t trow = static_cast<size_t>(row0 + tl), orow = trow * p.heads + h;
      const int col0 = v_first(pass0 + pi) * 64;
      float* const sums = s_max + (it & 1) * 2 * kRows + r;              // (last read before the last page's barrier)
      sums[hf * kRows] = l;
      meet();
      l = sums[0] + sums[kRows];
      meet();
      float inv = l > 0.f ? 1.f / l : 0.f;
      if (p.nsplit == 1 && p.gate && !p.gate_elems && valid) inv *= sigmoid_f(p.gate[trow * p.ld_gate + h]);
      const float* ge = p.gate && p.gate_elems ? p.gate + trow * p.ld_gate + static_cast<size_t>(h) * p.vdim + col0 : nullptr;
#pragma unroll 1
      for (int c0 = hf * vn * 32; c0 < (hf + 1) * vn * 32; c0 += 32) {
        uint32_t o[32];
        tmem_ld_x32(o_tm + lane_base + c0, o);
        tc_wait_ld();
        if (valid && p.nsplit > 1) {
          float* dst = p.part_o + (orow * p.nsplit + sp) * p.vdim + col0 + c0;
#pragma unroll
          for (int i = 0; i < 32; i += 8)
            st32(dst + i, make_uint4(o[i], o[i + 1], o[i + 2], o[i + 3]), make_uint4(o[i + 4], o[i + 5], o[i + 6], o[i + 7]), a.wide_out);
        } else if (valid) {
          if (ge) {
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * sigmoid_f(ge[c0 + i]));
          }
          if (p.out_f32) {
            float* dst = reinterpret_cast<float*>(p.out) + orow * p.vdim + col0 + c0;
            auto four = [&](int i) {
              return make_uint4(__float_as_uint(__uint_as_float(o[i]) * inv), __float_as_uint(__uint_as_float(o[i + 1]) * inv),
                                __float_as_uint(__uint_as_float(o[i + 2]) * inv), __float_as_uint(__uint_as_float(o[i + 3]) * inv));
            };
#pragma unroll
            for (int i = 0; i < 32; i += 8) st32(dst + i, four(i), four(i + 4), a.wide_out);
          } else {
            __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.out) + orow * p.vdim + col0 + c0;
            auto eight = [&](int i) {
              auto two = [&](int k) { return pack16x2<true>(__uint_as_float(o[k]) * inv, __uint_as_float(o[k + 1]) * inv); };
              return make_uint4(two(i), two(i + 2), two(i + 4), two(i + 6));
            };
#pragma unroll
            for (int i = 0; i < 32; i += 16) st32(dst + i, eight(i), eight(i + 8), a.wide_out);
          }
        }
        __syncwarp();
      }
      if (p.nsplit > 1 && valid && col0 == 0 && hf == 0) {
        float* ml = p.part_ml + (orow * p.nsplit + sp) * 2;
        ml[0] = m_ref * kLn2;
        ml[1] = l;
      }
      tc_fence_before();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, a.tmem_cols);
  }
}

constexpr int kSmemMax = 227 * 1024, kBarBytes = 256 + 4 * kRows * 4;       // (and the rows' maxima)

// Sizes of one launch; false: the shape does not fit.
static bool plan(const AttnTcProblem& p, Args& a) {
  a.p = p;
  a.shared = p.v_cache == nullptr;
  a.group = p.heads / p.kv_heads;
  if (a.group > kRows || p.dim % 32 != 0 || p.dim < 64 || p.vdim % 64 != 0 || p.vdim <= 0) return false;
  if (a.shared && (p.vdim > p.dim || p.kv_heads != 1)) return false;
  a.tq = kRows / a.group;
  a.kblk = p.dim / 64;
  a.tail = (p.dim % 64) / 32;
  const int vb = p.vdim / 64;
  a.passes = (vb + 3) / 4;
  a.vblk = (vb + a.passes - 1) / a.passes;
  a.passes = (vb + a.vblk - 1) / a.vblk;
  const int last = vb - (a.passes - 1) * a.vblk;              // value blocks of the last pass: the most key blocks beside them
  a.v_stage = a.vblk * kBlk;
  a.k_stage = (a.shared ? a.kblk - last : a.kblk) * kBlk + a.tail * kTailBlk;
  const int tm_room = (512 - a.vblk * 64 - 96) / 32;          // query blocks that TMEM can hold
  // Latent rows want three V stages (a page's value blocks stay until P V, one page after S); queries move to TMEM until
  // that fits, and with the last one moved two stages have to do.
  const int want_v = a.shared ? 3 : 2;
  for (a.sv = want_v; a.sv >= 2; --a.sv)
    for (a.q_tm = 0; a.q_tm <= (a.shared ? std::min(tm_room, a.kblk) : 0); ++a.q_tm) {
      a.sk = 2;
      a.q_bytes = (a.kblk - a.q_tm) * kQBlk + a.tail * kQTail;
      const int rings = a.sk * a.k_stage + a.sv * a.v_stage;
      if (a.q_bytes + rings + kBarBytes > kSmemMax) continue;
      if (a.q_tm * kQBlk > rings) continue;
      const int cols = a.vblk * 64 + 96 + a.q_tm * 32;
      a.tmem_cols = cols <= 128 ? 128 : (cols <= 256 ? 256 : 512);
      return true;
    }
  return false;
}

static bool page_map(CUtensorMap* m, const void* base, int row, int heads, int box_cols, CUtensorMapSwizzle swz) {
  // the page count is not known here: block tables hold valid pages only, so the outer extent is left open
  const uint64_t dims[4] = {static_cast<uint64_t>(row), static_cast<uint64_t>(heads), kTok, 1u << 25};
  const uint64_t tok = static_cast<uint64_t>(row) * heads * 2;
  const uint64_t strides[3] = {static_cast<uint64_t>(row) * 2, tok, tok * kTok};
  const uint32_t box[4] = {static_cast<uint32_t>(box_cols), 1, kTok, 1}, es[4] = {1, 1, 1, 1};
  return encode_tensor_map(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, es, swz,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B) == CUDA_SUCCESS;
}

}  // namespace hat

bool attn_tc_takes(const AttnTcProblem& p) {
  hat::Args a;
  const uintptr_t ptrs = reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k_cache) |
                         reinterpret_cast<uintptr_t>(p.v_cache) | reinterpret_cast<uintptr_t>(p.out) |
                         reinterpret_cast<uintptr_t>(p.part_o);
  return (ptrs & 15) == 0 && p.scale > 0.f && hat::plan(p, a);
}

int attn_tc_splits(int T, int kv_heads, int vdim, int shared_kv, int window, int keep_first, int max_blocks) {
  // every row is a tile of its own (one token per sequence), or a few of one sequence share one; a block per pass
  const int passes = shared_kv ? (vdim + 255) / 256 : 1;
  const int blocks = T * kv_heads * passes;
  int n = ((shared_kv ? 1 : 2) * sm_count()) / std::max(1, blocks);
  int pages = max_blocks > 0 ? max_blocks : 1 << 20;
  if (window > 0) pages = std::min(pages, (window + std::max(keep_first, 0) + hat::kTok - 1) / hat::kTok + 1);
  // A part that holds no page still costs its block and its place in the merge (one row on 30 keys, 16 parts 12 us, one 9 us), and the
  // merge costs more than a few pages in turn once there are many rows: up to four pages make one part, or, in small steps, one
  // each, more pages two each.  us for one row on 700 keys, 16 heads of 64 with 16 parts of one page 16.8, with 6 of two pages 12.8;
  // 32 rows on a window of 100, 12 heads of 128 x 192: two parts 22.8, one 14.3; one row on 200 keys, 16 heads over 4: one part 13.9, four 12.4.
  // Never more parts for fewer pages: the workspace is sized without knowing max_blocks.
  if (pages <= 4 && blocks > 64) return 1;
  return std::max(1, std::min({n, pages <= 4 ? pages : std::max(4, (pages + 1) / 2), 16}));
}

void launch_attn_tc(const AttnTcProblem& p, cudaStream_t st) {
  using namespace hat;
  Args a;
  if (!plan(p, a)) {
    set_error(1, "attn_tc: shape not supported");
    return;
  }
  CUtensorMap kmap, tmap, vmap;
  bool ok = page_map(&kmap, p.k_cache, p.dim, p.kv_heads, 64, CU_TENSOR_MAP_SWIZZLE_128B);
  tmap = vmap = kmap;
  if (a.tail) ok = ok && page_map(&tmap, p.k_cache, p.dim, p.kv_heads, 32, CU_TENSOR_MAP_SWIZZLE_64B);
  if (!a.shared) ok = ok && page_map(&vmap, p.v_cache, p.vdim, p.v_heads, 64, CU_TENSOR_MAP_SWIZZLE_128B);
  a.err = wait_error_flag();
  if (!ok || !a.err) {
    set_error(2, "attn_tc: cuTensorMapEncodeTiled failed");
    return;
  }
  const int smem = a.q_bytes + a.sk * a.k_stage + a.sv * a.v_stage + kBarBytes;
  const int tiles = (p.T + a.tq - 1) / a.tq + p.num_seqs;
  // all passes in one block (Q is staged once) where that still gives every SM two blocks; otherwise a block per pass
  a.page_ref = attn_few_rows(p.T);
  a.ppc = p.nsplit == 1 && tiles * p.kv_heads >= 2 * sm_count() ? a.passes : 1;
  const dim3 grid(tiles, p.kv_heads, p.nsplit * (a.passes / a.ppc));
  a.by_group = (65536 + a.group - 1) / a.group;
  a.wide_q = (reinterpret_cast<uintptr_t>(p.q) & 31) == 0;
  a.wide_out = ((reinterpret_cast<uintptr_t>(p.out) | reinterpret_cast<uintptr_t>(p.part_o)) & 31) == 0;
  const bool cap = p.softcap > 0.f, bias = p.slopes || p.dist_bias;
  auto kern = cap ? (bias ? attn_tc_kernel<true, true> : attn_tc_kernel<true, false>)
                  : (bias ? attn_tc_kernel<false, true> : attn_tc_kernel<false, false>);
  static OncePerDevice sized[4];
  if (!allow_smem(sized[cap * 2 + bias], kern, kSmemMax)) return;
  kern<<<grid, kThreads, smem, st>>>(kmap, tmap, vmap, a);
  B200_CUDA_LAUNCH_CHECK();
}

}  // namespace b200
