"""The count-1 flag told from the words around a one-group run (single_flag,
wah_core.cuh), against the walk's step states, on the CPU
(tests/group_model.cpp over the product header)."""
import ctypes
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("group") / "libgroup.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", out,
                    os.path.join(ROOT, "tests", "group_model.cpp")], check=True)
    lib = ctypes.CDLL(out)
    lib.group_model_mismatches.restype = ctypes.c_long
    return lib


@pytest.mark.parametrize("op", range(4))
def test_single_group_runs(model, op):
    assert model.group_model_mismatches(op, 17 + op, ctypes.c_long(60_000)) == 0
