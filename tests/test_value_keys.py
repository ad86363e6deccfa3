"""Value keys (wah_keys.h) against the double comparison they stand for, on
the CPU: every pair of comparisons, bounds on, between and beyond the values,
infinities, NaN and both zeros, for each column type."""
import ctypes
import itertools
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SRC = r'''
#include "wah_keys.h"
using namespace wah;
extern "C" int in_range(uint32_t bits, uint32_t vtype, uint32_t lop, double lo, uint32_t rop, double hi) {
    uint32_t k, s;
    if (!key_range(vtype, lop, lo, rop, hi, k, s)) return 0;
    return value_key(bits, key_map(vtype)) - k <= s;
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("keys")
    (d / "keys.cpp").write_text(SRC)
    out = str(d / "libkeys.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "libfastlib_b200", "csrc"),
                    "-o", out, str(d / "keys.cpp")], check=True)
    L = ctypes.CDLL(out)
    L.in_range.argtypes = [ctypes.c_uint32, ctypes.c_uint32, ctypes.c_uint32, ctypes.c_double, ctypes.c_uint32,
                           ctypes.c_double]
    return L


@pytest.mark.parametrize("vtype,dtype", [(0, np.uint32), (1, np.float32), (2, np.int32)])
def test_same_as_double_comparison(lib, vtype, dtype):
    rng = np.random.default_rng(vtype)
    if vtype == 1:
        vals = np.array([0.0, -0.0, 1e-45, -1e-45, 1.0, -1.0, 0.1, 3.4e38, -3.4e38, np.inf, -np.inf, np.nan, 7.25, 16777216.0],
                        np.float32)
        vals = np.concatenate([vals, rng.normal(size=30).astype(np.float32), [np.float32(-np.nan)]])
        bounds = [0.0, -0.0, 0.1, 0.1 + 1e-12, 1.0, -1.0, 1e-50, -1e-50, 3.5e38, -3.5e38, np.inf, -np.inf, np.nan,
                  16777216.5, 16777217.0] + [float(v) for v in vals[14:20]] + [float(v) + 1e-9 for v in vals[14:18]]
    else:
        info = np.iinfo(dtype)
        vals = np.concatenate([np.array([info.min, info.min + 1, 0, 1, 2, 50, info.max - 1, info.max], dtype),
                               rng.integers(info.min, info.max, 20, dtype=np.int64).astype(dtype)])
        bounds = [float(info.min), float(info.min) - 0.5, -0.0, 0.0, 0.5, 1.0, 1.5, 50.0, 49.999, float(info.max),
                  float(info.max) + 1.0, 1e300, -1e300, np.inf, -np.inf, np.nan] + [float(v) for v in vals[8:12]]
    bits = vals.view(np.uint32)
    for lop, rop in itertools.product(range(3), range(3)):
        if lop == 0 and rop == 0:
            continue  # no bound: no edge rows to compare
        for lo, hi in itertools.product(bounds if lop else [0.0], bounds if rop else [0.0]):
            for v, b in zip(vals, bits):
                x = float(v)
                want = (lop == 0 or (lo < x if lop == 1 else lo <= x)) and (rop == 0 or (x < hi if rop == 1 else x <= hi))
                assert bool(lib.in_range(int(b), vtype, lop, lo, rop, hi)) == want, (x, lop, lo, rop, hi)
