"""A batched plan of dependent calls beside a kernel that keeps most of the GPU."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
def test_dependent_plan_beside_a_resident_kernel(gpu_built, tmp_path):
    exe = str(tmp_path / "resident_check")
    lib = os.path.join(gpu_built.PKG, "build")
    nvcc = os.path.join(os.environ.get("CUDA", "/usr/local/cuda"), "bin", "nvcc")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O2", "-rdc=true",
                        "-Xcudafe", "--diag_suppress=177", "-I", os.path.join(ROOT, "include"),
                        "-I", os.path.join(ROOT, "include", "gpumpi"),
                        os.path.join(ROOT, "tests", "native", "resident_check.cu"), "-o", exe, "-L", lib, "-lgpumpi",
                        "-Xlinker", "-rpath", "-Xlinker", lib], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
