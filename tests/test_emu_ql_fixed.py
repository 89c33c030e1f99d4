"""The Hermitian solver's fixed-point QL kernel (stablercwa_gb300/csrc/eig_fixed.cuh) compiled for the host: every
eigenvalue of lossless grating layers (orders 2 to 301) against bisection in long double, within 2^-54 of Gershgorin's
bound, one FP64 rounding of an entry of that size (tests/emu/warp/ql_fixed_emu.cpp)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_fixed_point_ql_eigenvalues(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = tmp_path / "ql_fixed_emu"
    build = subprocess.run([cxx, "-O2", "-std=c++20", "-I", os.path.join(HERE, "emu", "warp"), "-o", str(exe),
                            os.path.join(HERE, "emu", "warp", "ql_fixed_emu.cpp")], capture_output=True, text=True, timeout=300)
    assert build.returncode == 0, build.stderr[-2000:]
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and run.stdout.strip().endswith("OK"), run.stdout[-3000:]
    assert run.stdout.count("pass ") == 6
