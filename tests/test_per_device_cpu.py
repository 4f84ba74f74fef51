"""Once per device: kernel attributes that one device has say nothing about the next, and a failure is tried again."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "vllm_rs_b200" / "csrc"
PROGRAM = r'''
#include <initializer_list>
#include "host/per_device.hpp"
int main() {
  b200::OncePerDevice once, other;
  int calls[70] = {}, fail = 1;
  auto set = [&](int dev) { return once(dev, [&] { ++calls[dev < 0 ? 69 : dev]; return dev == 2 && fail ? 7 : 0; }); };
  for (int round = 0; round < 2; ++round)
    for (int dev : {0, 1, 63}) if (set(dev) != 0) return 1;
  if (calls[0] != 1 || calls[1] != 1 || calls[63] != 1) return 2;
  if (set(2) != 7 || set(2) != 7 || calls[2] != 2) return 3;      // a failure is told, and tried again
  fail = 0;
  if (set(2) != 0 || set(2) != 0 || calls[2] != 3) return 4;
  if (set(64) != 0 || set(64) != 0 || calls[64] != 2 || set(-1) != 0) return 5;      // not counted: set every time
  int n = 0;
  if (other(0, [&] { return ++n, 0; }) != 0 || n != 1) return 6;  // another kernel's
  return 0;
}
'''


def test_once_per_device(tmp_path):
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


@pytest.mark.parametrize("name", ["paged_attn_tc.cu", "moe_tc.cu", "linear_recurrence.cu"])
def test_no_attribute_is_set_once_per_process(name):
    """The persistent kernels of the hybrid decoders ask for their shared memory on every device that runs them."""
    src = (CSRC / name).read_text()
    assert "allow_smem(" in src and "cudaFuncSetAttribute" not in src
