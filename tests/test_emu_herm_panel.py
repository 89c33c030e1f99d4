"""The blocked Hermitian reduction's fixed-point panel (stablercwa_gb300/csrc/herm_fixed.cuh) compiled for the host and run
through the warp-level emulation of tests/emu/warp/: d and e against the FP64 panel's, and the same bits whatever the order
of a warp's lanes between barriers and whatever the workspace held, also where columns need no reflector."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_fixed_point_panel_in_emulation(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = tmp_path / "herm_panel_emu"
    build = subprocess.run([cxx, "-O2", "-std=c++20", "-I", os.path.join(HERE, "emu", "warp"), "-o", str(exe),
                            os.path.join(HERE, "emu", "warp", "herm_panel_emu.cpp")], capture_output=True, text=True, timeout=300)
    assert build.returncode == 0, build.stderr[-2000:]
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and run.stdout.strip().endswith("OK"), run.stdout[-3000:]
    assert run.stdout.count("pass ") == 25
