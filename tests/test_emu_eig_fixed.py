"""The fixed-point general eigensolver's kernels (stablercwa_gb300/csrc/eig_fixed.cuh) compiled for the host and
run through a warp-level emulation of the CUDA primitives they use (tests/emu/warp/): the rotation coefficients
on 200,000 triples against long double (within 2^-57, a sixteenth of FP64's rounding), and whole solves on random
matrices of orders 2..97 (the edges of the 32-column blocks and tiles), matrices scaled by 1e-30 and 1e40,
absorbing and lossless grating layers up to order 161, diagonal and triangular matrices with repeated entries,
blocks of very different size, and what is left to the FP64 kernels (zero, non-finite and extreme matrices, one
that needs an exceptional shift beyond the scale); and the Hermitian solver's pieces (the reduction, the QL
iteration, both sets of rotations) on random Hermitian, lossless grating, diagonal and Wilkinson W+ matrices.
Orthogonality, Schur residual and eigenpair residuals are held
to 1e-13, the bound of the FP64 solver's tests."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_fixed_point_eigensolver_in_emulation(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = tmp_path / "eig_fixed_emu"
    build = subprocess.run([cxx, "-O2", "-std=c++20", "-I", os.path.join(HERE, "emu", "warp"), "-o", str(exe),
                            os.path.join(HERE, "emu", "warp", "eig_fixed_emu.cpp")], capture_output=True, text=True, timeout=300)
    assert build.returncode == 0, build.stderr[-2000:]
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=900)
    assert run.returncode == 0 and run.stdout.strip().endswith("OK"), run.stdout[-3000:]
    assert run.stdout.count("pass ") == 41
