"""The order in which the truncation kernels take singular values, compiled for the host: positions
counted with it are a permutation for any values (NaN and infinities among them), and for numbers the
descending order with ties by index."""
import itertools
import os
import subprocess

import numpy as np
import pytest
from conftest import ROOT

PROGRAM = r"""
#include "sigma_order.h"
extern "C" void positions(const double* s, int k, int* pos) {
  for (int j = 0; j < k; ++j) {
    pos[j] = 0;
    for (int i = 0; i < k; ++i) pos[j] += hmatb200::sigma_before(s[i], i, s[j], j);
  }
}
"""


@pytest.fixture(scope="module")
def positions(tmp_path_factory):
    import ctypes
    d = tmp_path_factory.mktemp("sigma")
    (d / "p.cpp").write_text(PROGRAM)
    so = str(d / "p.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, "hmat-oss_b200", "csrc"),
                    str(d / "p.cpp"), "-o", so], check=True)
    f = ctypes.CDLL(so).positions

    def run(values):
        s = np.array(values, dtype=np.float64)
        out = np.empty(len(s), dtype=np.int32)
        f(s.ctypes.data_as(ctypes.c_void_p), len(s), out.ctypes.data_as(ctypes.c_void_p))
        return out
    return run


def test_positions_are_a_permutation(positions):
    pool = [float("nan"), float("inf"), 0.0, 2.5, 1.0]
    for k in range(1, 6):
        for v in itertools.product(pool, repeat=k):
            assert sorted(positions(v)) == list(range(k)), v


def test_numbers_in_descending_order_ties_by_index(positions):
    rng = np.random.default_rng(0)
    for k in (1, 2, 17, 64, 128):
        v = rng.integers(0, max(2, k // 2), k).astype(float)
        order = np.argsort(-v, kind="stable")
        want = np.empty(k, dtype=int)
        want[order] = np.arange(k)
        assert np.array_equal(positions(v), want)
