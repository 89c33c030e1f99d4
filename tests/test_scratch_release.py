"""The batched solvers give their scratch back when one of their allocations fails: the built objects are linked with a
replaced allocator (tests/emu/alloc/scratch_release.cu) in which the k-th allocation fails, for every k. Runs without a
device, and hides any there is."""
import glob
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
WRAPPED = ["cudaMallocAsync", "cudaFreeAsync", "cudaLaunchKernel", "cudaGetLastError", "cudaFuncSetAttribute", "cudaGetDevice",
           "cudaMalloc", "cudaMemset", "cudaMemsetAsync", "cudaMemcpy2DAsync"]


def test_scratch_is_released_when_an_allocation_fails(tmp_path):
    from stablercwa_gb300 import build
    nvcc = build._nvcc()
    if shutil.which(nvcc) is None:
        pytest.skip("no nvcc")
    build.build()
    objects = sorted(glob.glob(os.path.join(build.BUILD, "*.o")))
    if not objects:
        pytest.skip("the engine's objects are not there")
    exe = tmp_path / "scratch_release"
    wraps = [x for name in WRAPPED for x in ("-Xlinker", f"--wrap={name}")]
    made = subprocess.run([nvcc, *build.ARCH, "-std=c++17", "-diag-suppress", "177", "-o", str(exe),
                           os.path.join(HERE, "emu", "alloc", "scratch_release.cu"), *objects, "-lpthread", *wraps],
                          capture_output=True, text=True, timeout=600)
    assert made.returncode == 0, made.stderr[-2000:]
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300,
                         env=dict(os.environ, CUDA_VISIBLE_DEVICES=""))
    assert run.returncode == 0 and run.stdout.strip().endswith("OK"), run.stdout[-3000:]
