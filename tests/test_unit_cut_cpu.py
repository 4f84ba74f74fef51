"""The cut of a quantised product's units over blocks (csrc/host/unit_cut.hpp), beside integer division."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "vllm_rs_b200" / "csrc"
PROGRAM = r'''
#include <cstdio>
#include <initializer_list>
#include "host/unit_cut.hpp"
using namespace b200;
// 0: as it must be; -1: the size is refused
static int check(int K, int N, int most) {
  const int tiles = N / 128, U = K / 128;
  UnitCut c;
  const int grid = cut_units(tiles, U, most, 2, c);
  if (grid == 0) return -1;
  const int total = tiles * U;
  const UnitDiv by_U = unit_div(U);
  if (grid > most || c.start(0) != 0 || c.start(grid) != total) return 1;
  for (int i = 0; i < grid; ++i) {
    const int u0 = c.start(i), u1 = c.start(i + 1);
    if (u1 <= u0) return 2;                                                        // no block without a unit
    if (c.block_of(u0) != i || c.block_of(u1 - 1) != i) return 3;
    if (by_U(u0) != u0 / U || by_U(u1 - 1) != (u1 - 1) / U) return 4;
    if (!c.whole && u0 / U != (u1 - 1) / U) return 5;                              // cut alike: no block has two tiles
  }
  for (int t = 0; t < tiles; ++t) {                                                // who meets for a tile
    const int b0 = c.block_of(t * U), b1 = c.block_of(t * U + U - 1);
    if (b0 < 0 || b1 >= grid || b0 > b1) return 6;
    if (c.start(b0) > t * U || c.start(b0 + 1) <= t * U || c.start(b1) > t * U + U - 1 || c.start(b1 + 1) < t * U + U) return 7;
  }
  return 0;
}
int main() {
  long taken = 0, large = 0, refused = 0;
  for (int most : {148, 264, 296})
    for (int K = 128; K <= 65536; K += K < 2048 ? 128 : K < 16384 ? 1408 : 3712)
      for (int N = 128; N <= 524288; N += N < 4096 ? 384 : N < 65536 ? 2432 : 29696) {
        const int e = check(K, N, most);
        if (e > 0) return std::printf("K %d N %d blocks %d: %d\n", K, N, most, e), 1;
        taken += e == 0;
        refused += e < 0;
        large += e == 0 && static_cast<long>(K / 128) * (N / 128) > 65536;
      }
  const int sizes[][2] = {{34944, 30848}, {35584, 30720}, {32768, 32896}, {65536, 16512}, {128, 524288}, {28672, 8192}};
  for (auto& s : sizes)
    if (check(s[0], s[1], 296) != 0) return std::printf("K %d N %d\n", s[0], s[1]), 1;
  std::printf("%ld %ld %ld\n", taken, large, refused);
  return taken > 5000 && large > 500 ? 0 : 2;
}
'''


def test_cut_is_exact_at_every_size(tmp_path):
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
