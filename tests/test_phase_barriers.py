"""The block-wide barriers between the phases of the FP64 characteristic
kernels (csrc/physics_exact.cuh char_pair): every thread of a block meets
every one, also past the range and at nodes without a face, counted on the
host (tests/cpp/phase_barrier_check.cpp)."""
from __future__ import annotations

import pathlib
import shutil
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
CSRC = ROOT / "high-order-accurate-cfd-solver-code-for-heterogenous-hardware-cpu-and-gpgpu-_gb300" / "csrc"


def test_every_thread_meets_every_barrier(pkg, tmp_path):
    from cfd_gb300 import build
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    cuda = pathlib.Path(build.nvcc()).resolve().parents[1] / "include"
    exe = tmp_path / "phase_barrier_check"
    subprocess.run([cxx, "-std=c++17", "-O1", "-ffp-contract=off", "-I", str(cuda), "-I", str(ROOT / "include"),
                    "-I", str(CSRC), str(ROOT / "tests" / "cpp" / "phase_barrier_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
