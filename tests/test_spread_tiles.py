"""The tile lists of launch-ordered plans, checked on the CPU.

The host code that cuts collective calls into tiles (csrc/spread.cu, in
libgpumpi.so) needs no GPU: a small program links it, emulates the accesses of
every tile for random calls and reports reads outside the source buffers,
destination bytes not written exactly once, misaligned units and rows that do
not fit the ring.
"""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "dphpc-project_gb300")


@pytest.fixture(scope="module")
def spread_check(tmp_path_factory):
    lib = os.path.join(PKG, "build")
    if not os.path.exists(os.path.join(lib, "libgpumpi.so")):
        subprocess.run(["make", "-C", PKG, "-j8", "build/libgpumpi.so"], check=True, capture_output=True)
    exe = tmp_path_factory.mktemp("spread") / "spread_check"
    nvcc = os.path.join(os.environ.get("CUDA", "/usr/local/cuda"), "bin", "nvcc")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O2", "-rdc=true",
                        "-Xcudafe", "--diag_suppress=177", "-I", os.path.join(ROOT, "include"),
                        "-I", os.path.join(ROOT, "include", "gpumpi"), "-I", os.path.join(PKG, "csrc"),
                        os.path.join(ROOT, "tests", "native", "spread_check.cu"), "-o", str(exe), "-L", lib, "-lgpumpi",
                        "-Xlinker", "-rpath", "-Xlinker", lib], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return str(exe)


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_tiles_stay_in_bounds_and_write_every_byte_once(spread_check, seed):
    r = subprocess.run([spread_check, str(seed), "1000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr
    assert "bad 0" in r.stdout
