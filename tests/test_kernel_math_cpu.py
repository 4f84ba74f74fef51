"""Approximations that kernels use, from their constants in the source, against 64 bits."""
import ctypes
import re
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "vllm_rs_b200" / "csrc"


def test_tanh_fit():
    src = (CSRC / "paged_attn_tc.cu").read_text()
    top = float(re.search(r"kTanhMax = ([0-9.]+)f", src).group(1))
    c = [np.float64(np.float32(re.search(rf"kT{i} = (-?[0-9.]+)f", src).group(1))) for i in range(6)]
    said = float(re.search(r"relative error ([0-9.e-]+) before rounding", src).group(1))
    y = np.linspace(1e-6, top, 400001)
    err = np.abs(y * np.polynomial.polynomial.polyval(y * y, c) / np.tanh(y) - 1).max()
    assert 0.5 * said < err <= said


def test_parts_never_grow_with_fewer_pages():
    """The workspace of split keys is sized for the longest context; a rule restated from the source has to keep to it."""
    src = (CSRC / "paged_attn_tc.cu").read_text()
    body = src[src.index("int attn_tc_splits("):]
    body = body[:body.index("\n}\n")]
    assert "pages <= 4 && blocks > 64" in body and "pages <= 4 ? pages : std::max(4, (pages + 1) / 2), 16" in body

    def parts(n, blocks, pages):
        if pages <= 4 and blocks > 64:
            return 1
        return max(1, min(n, pages if pages <= 4 else max(4, (pages + 1) // 2), 16))
    for n in range(1, 20):
        for blocks in (1, 64, 65, 500):
            got = [parts(n, blocks, p) for p in range(1, 70)]
            assert got == sorted(got)


def test_swizzled_places_begin_the_shared_memory():
    """attn_tc_kernel has no room for a round-up to its swizzles' 1024 bytes: dynamic shared memory begins on them as long as there is
    no static one in front."""
    src = (CSRC / "paged_attn_tc.cu").read_text()
    assert re.findall(r"^.*__shared__.*$", src, re.M) == ["  extern __shared__ __align__(1024) uint8_t smem[];"]


@pytest.mark.parametrize("T,ff,K,own", [(3001, 5632, 2048, True), (1000, 5632, 2048, True), (256, 5632, 2048, False), (300, 512, 2048, False),
                                        (3001, 512, 2048, False), (300, 11008, 2048, False), (512, 11008, 2048, True),
                                        (1000, 5632, 1024, False), (3001, 5632, 1024, True), (1500, 2816, 4096, True), (129, 8, 64, False)])
def test_gated_rows_take_the_faster_way(T, ff, K, own):
    """Sizes whose times stand on the one side or the other, by 5 % at least, of the library's and a pass over its results."""
    from vllm_rs_b200 import _lib
    pays = getattr(_lib.lib(), "_ZN4b20016dense_gated_paysEiiii")
    pays.restype = ctypes.c_bool
    assert pays(T, ff, K, 74) == own
