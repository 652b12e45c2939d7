"""Quotients and square roots on the integer pipe (csrc/exact_int.cuh) from
seeds as far off as the device's approximations may be
(tests/cpp/seed_bound_check.cpp)."""
from __future__ import annotations

import pathlib
import shutil
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
CSRC = ROOT / "high-order-accurate-cfd-solver-code-for-heterogenous-hardware-cpu-and-gpgpu-_gb300" / "csrc"


def test_results_hold_for_every_seed_in_the_documented_bound(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "seed_bound_check"
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(CSRC),
                    str(ROOT / "tests" / "cpp" / "seed_bound_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
