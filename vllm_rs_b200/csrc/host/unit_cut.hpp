// How the units (tile of 128 channels x 128 K) of a quantised product are cut over the blocks of a launch: made on the host,
// looked up by the kernel.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define B200_CUT_FN __host__ __device__ __forceinline__
#else
#define B200_CUT_FN inline
#endif

namespace b200 {

// x / d by one multiplication: m = ceil(2^32 / d) is exact for x * d < 2^32; d = 1: m = 0.
struct UnitDiv {
  uint32_t m;
  B200_CUT_FN int operator()(int x) const {
#ifdef __CUDA_ARCH__
    return m ? static_cast<int>(__umulhi(x, m)) : x;
#else
    return m ? static_cast<int>(static_cast<uint64_t>(static_cast<uint32_t>(x)) * m >> 32) : x;
#endif
  }
};
inline UnitDiv unit_div(int d) { return UnitDiv{d > 1 ? static_cast<uint32_t>(((1ull << 32) + d - 1) / d) : 0u}; }

// Every `period` units (a tile, or, where `whole`, all there are) go to `parts` blocks, of which the first `rest` have share + 1
// units and the others `share`.
struct UnitCut {
  int period, parts, share, rest, whole;
  UnitDiv by_period, by_parts, by_share, by_more;
  // first unit of block i (of the block past the last: the number of units)
  B200_CUT_FN int start(int i) const {
    const int q = whole ? 0 : by_parts(i), j = i - q * parts;
    return q * period + j * share + (j < rest ? j : rest);
  }
  B200_CUT_FN int block_of(int unit) const {
    const int q = whole ? 0 : by_period(unit), j = unit - q * period, head = rest * (share + 1);
    return q * parts + (j < head ? by_more(j) : rest + by_share(j - head));
  }
};

// tiles x U units in `parts` parts per tile, or (0) in ranges cut anywhere for `grid` blocks.  Returns the number of blocks; 0 where a
// division would not be exact.
inline int cut_parts(int tiles, int U, int parts, int grid, UnitCut& c) {
  const int64_t all = static_cast<int64_t>(tiles) * U;
  if (all >= int64_t{1} << 31) return 0;
  const int total = static_cast<int>(all);
  c.whole = !parts;
  if (!c.whole) grid = tiles * parts;
  if (grid > total) grid = total;
  c.period = c.whole ? total : U;
  c.parts = c.whole ? grid : parts;
  c.share = c.period / c.parts;
  c.rest = c.period % c.parts;
  // What is divided: units by U (by the kernel, and as `period` where tiles are cut alike); places in a period by share and share + 1;
  // blocks, up to `grid`, by parts.  A division by all units, which is 0 for every unit, would not be exact past 65536 of them.
  const int64_t widest = U > c.share + 1 ? U : c.share + 1;
  if (total * widest >= int64_t{1} << 31 || static_cast<int64_t>(grid) * c.parts >= int64_t{1} << 31) return 0;
  c.by_period = unit_div(c.period);
  c.by_parts = unit_div(c.parts);
  c.by_share = unit_div(c.share);
  c.by_more = unit_div(c.share + 1);
  return grid;
}

// The cut of tiles x U units for at most `most` blocks of `groups` groups each, of which every one takes a unit in turn.
// Every tile in the same number of parts, at most eight, where that leaves few blocks out: no block has then two tiles.
// 4096 x 4096, one token: 8 parts 5.4 us, 4 parts 7.1.  Otherwise ranges cut anywhere.
inline int cut_units(int tiles, int U, int most, int groups, UnitCut& c) {
  if (static_cast<int64_t>(tiles) * U >= int64_t{1} << 31) return 0;
  int splits = most / tiles;
  if (splits > U / groups) splits = U / groups;
  if (splits > 8) splits = 8;
  const bool even = splits >= 1 && (tiles * splits * 100 >= most * 85 || tiles * U < most * groups || tiles * 8 < most);
  return cut_parts(tiles, U, even ? splits : 0, most, c);
}

}  // namespace b200
