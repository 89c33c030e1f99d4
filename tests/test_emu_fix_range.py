"""Which matrices the fixed-point eigensolvers leave to the FP64 kernels (fix_range_kernel, fix_keeps_fp64 in
stablercwa_gb300/csrc/eig_fixed.cuh), compiled for the host and run through the warp-level emulation of tests/emu/warp/:
matrices whose small eigenvalues FP64 keeps relative to themselves stay there, layer matrices do not."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_range_of_the_fixed_point_solvers(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = tmp_path / "range_emu"
    build = subprocess.run([cxx, "-O2", "-std=c++20", "-I", os.path.join(HERE, "emu", "warp"), "-o", str(exe),
                            os.path.join(HERE, "emu", "warp", "range_emu.cpp")], capture_output=True, text=True, timeout=300)
    assert build.returncode == 0, build.stderr[-2000:]
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and run.stdout.strip().endswith("OK"), run.stdout[-3000:]
