"""Products, quotients and square roots on the integer pipe
(csrc/exact_int.cuh): the bits of the host's IEEE operations, on operands of
every class (tests/cpp/exact_int_check.cpp).  The device's results are
compared with its own instructions by cfd_probe_emu64 (test_gpu_emu64.py)."""
from __future__ import annotations

import pathlib
import shutil
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
CSRC = ROOT / "high-order-accurate-cfd-solver-code-for-heterogenous-hardware-cpu-and-gpgpu-_gb300" / "csrc"


@pytest.mark.parametrize("seed", [1, 20261205])
def test_integer_pipe_results_are_ieee(tmp_path, seed):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "exact_int_check"
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(CSRC),
                    str(ROOT / "tests" / "cpp" / "exact_int_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe), "2000000", str(seed)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
