"""The server's charge against what admitted batches take (wah_budget.h), on
the CPU."""
import ctypes
import os
import subprocess

from conftest import ROOT


def test_batches_stay_within_the_budget(tmp_path):
    out = str(tmp_path / "libbudget.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-o", out,
                    os.path.join(ROOT, "tests", "budget_model.cpp")], check=True)
    assert ctypes.CDLL(out).budget_model(5, 3000) == 0
