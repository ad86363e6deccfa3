"""The block pool behind the device and pinned allocations (wah_pool.h), on
the CPU over a driver that counts and can run out of memory."""
import ctypes
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("pool") / "libpool.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-o", out,
                    os.path.join(ROOT, "tests", "pool_model.cpp")], check=True)
    return ctypes.CDLL(out)


@pytest.mark.parametrize("seed", range(4))
def test_pool(model, seed):
    assert model.pool_model(seed, 4000) == 0
