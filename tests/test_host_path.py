"""Host side of the collective API on a fake CUDA runtime.

The objects of libgpumpi.so are linked with a CUDA runtime that runs on the CPU
and records what is enqueued on which stream (tests/native/fake_cuda.h), so the
order of copies and launches, allocations and error paths are tested without a
GPU and without a GPU fault.
"""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "dphpc-project_gb300")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    subprocess.run(["make", "-C", PKG, "-j8", "build/libgpumpi.so"], check=True, capture_output=True)
    build = os.path.join(PKG, "build")
    names = ("rt_core p2p coll ops dispatch api_p2p api_coll api_comm gmalloc libc host serve cluster server "
             "capi_coll spread capi_heap tune")
    objects = [os.path.join(build, n + ".o") for n in names.split()]
    cuda = os.environ.get("CUDA", "/usr/local/cuda")
    nvcc = [os.path.join(cuda, "bin", "nvcc"), "-gencode", "arch=compute_103a,code=sm_103a"]
    native = os.path.join(ROOT, "tests", "native")
    tmp = tmp_path_factory.mktemp("host_path")
    exe, fake, main, link = (str(tmp / f) for f in ("host_path_check", "fake.o", "main.o", "link.o"))
    for cmd in (["g++", "-std=c++17", "-O1", "-I", os.path.join(cuda, "include"), "-c",
                 os.path.join(native, "fake_cuda.cpp"), "-o", fake],
                [*nvcc, "-std=c++17", "-O1", "-rdc=true", "-Xcudafe", "--diag_suppress=177",
                 "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "include", "gpumpi"),
                 "-I", os.path.join(PKG, "csrc"), "-c", os.path.join(native, "host_path_check.cu"), "-o", main],
                [*nvcc, "-dlink", main, *objects, "-o", link],
                # no scenario makes the runtime calls that the fake one does not have
                ["g++", main, link, *objects, fake, "-lpthread", "-Wl,--unresolved-symbols=ignore-all", "-o", exe]):
        r = subprocess.run(cmd, capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr
    return exe


@pytest.mark.parametrize("scenario", ["tables", "uploaded", "retry", "order", "turns", "first_calls", "captured",
                                      "tuner_file", "one_shot_calls", "images", "errors", "levels", "random_levels",
                                      "long_plans", "devices", "failed_plans"])
def test_host_path(check, scenario):
    r = subprocess.run([check, scenario], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr
