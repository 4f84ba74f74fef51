"""Approximations that kernels use, from their constants in the source, against 64 bits."""
import re
from pathlib import Path

import numpy as np

CSRC = Path(__file__).resolve().parent.parent / "vllm_rs_b200" / "csrc"


def test_tanh_fit():
    src = (CSRC / "paged_attn_tc.cu").read_text()
    top = float(re.search(r"kTanhMax = ([0-9.]+)f", src).group(1))
    c = [np.float64(np.float32(re.search(rf"kT{i} = (-?[0-9.]+)f", src).group(1))) for i in range(6)]
    said = float(re.search(r"relative error ([0-9.e-]+) before rounding", src).group(1))
    y = np.linspace(1e-6, top, 400001)
    err = np.abs(y * np.polynomial.polynomial.polyval(y * y, c) / np.tanh(y) - 1).max()
    assert 0.5 * said < err <= said
