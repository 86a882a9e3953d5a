"""Tile lists on the CPU: exact cover of every destination, up to the most ranks that tiles take.

tests/native/spread_cover.cu emulates the accesses of every tile.  The named
calls are those whose sizes the GPU tests use to reach a form of tiles: a
threshold that moves does not silently drop their coverage.
"""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "dphpc-project_gb300")
OPS = {"bcast": 1, "reduce": 2, "allreduce": 3, "alltoall": 4, "allgather": 5}
TYPES = {"i1": (6, 1), "u1": (29, 1), "i2": (1, 2), "i4": (2, 4), "f4": (12, 4), "f8": (13, 8)}


@pytest.fixture(scope="module")
def cover(tmp_path_factory):
    subprocess.run(["make", "-C", PKG, "-j8", "build/libgpumpi.so"], check=True, capture_output=True)
    lib = os.path.join(PKG, "build")
    exe = str(tmp_path_factory.mktemp("cover") / "spread_cover")
    nvcc = os.path.join(os.environ.get("CUDA", "/usr/local/cuda"), "bin", "nvcc")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O2", "-rdc=true",
                        "-Xcudafe", "--diag_suppress=177", "-I", os.path.join(ROOT, "include"),
                        "-I", os.path.join(ROOT, "include", "gpumpi"), "-I", os.path.join(PKG, "csrc"),
                        os.path.join(ROOT, "tests", "native", "spread_cover.cu"), "-o", exe, "-L", lib, "-lgpumpi",
                        "-Xlinker", "-rpath", "-Xlinker", lib], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return exe


def test_random_calls_are_covered_exactly_once(cover):
    forms = set()
    for seed in (1, 2, 3):
        r = subprocess.run([cover, "random", str(seed), "900"], capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout[-3000:]
        forms |= set(r.stdout.split("forms ")[1].split())
    assert forms - {"rows-many"} == {"fan", "copy", "chunks", "gather", "stream", "rows", "passes", "move-alltoall",
                                     "move-fan"}


# (call, ranks, elements, type, skew) -> form of its tiles, alone in its level
FORMS = [
    ("allreduce", 256, 60001, "f8", 1, "gather"), ("allreduce", 257, 500, "f8", 0, "gather"),
    ("allreduce", 257, 20000, "f8", 0, "passes"), ("allreduce", 257, 20001, "f8", 1, "passes"),
    ("reduce", 1024, 60000, "f8", 0, "passes"), ("reduce", 1024, 60001, "f8", 1, "passes"),
    ("allreduce", 512, 20001, "i4", 1, "passes"), ("allreduce", 640, 700000, "u1", 0, "passes"),
    ("allreduce", 640, 700001, "u1", 1, "rows-many"), ("allreduce", 257, 160003, "f8", 1, "rows-many"),
    ("allreduce", 769, 165000, "f8", 0, "rows-many"), ("allreduce", 2048, 130001, "i4", 1, "passes"),
    ("allreduce", 4, 1000000, "f8", 0, "stream"), ("allreduce", 4, 1000001, "f8", 1, "rows"),
    ("reduce", 64, 62497, "f8", 1, "gather"), ("reduce", 64, 70001, "f8", 1, "rows"),
    ("allreduce", 20, 600001, "i4", 1, "rows"),
    ("bcast", 16, 750000, "f8", 0, "move-fan"), ("bcast", 16, 750001, "f8", 1, "move-fan"),
    ("bcast", 16, 6000001, "u1", 1, "move-fan"), ("allgather", 100, 1000, "f8", 0, "move-fan"),
    ("allgather", 100, 1001, "f8", 1, "move-fan"), ("allgather", 100, 8001, "u1", 1, "move-fan"),
    ("reduce", 256, 126952, "f8", 0, "rows"), ("reduce", 256, 126953, "f8", 1, "rows"),
    ("reduce", 256, 1015624, "u1", 0, "rows"), ("allreduce", 160, 812500, "u1", 0, "rows"),
    ("allreduce", 256, 97656, "f8", 0, "rows"), ("reduce", 320, 101560, "f8", 0, "rows-many"),
    ("allreduce", 17, 2000001, "i4", 1, "rows"), ("reduce", 512, 97657, "f8", 1, "rows-many"),
    ("alltoall", 128, 1524, "f8", 0, "copy"), ("alltoall", 31, 60000, "i4", 0, "copy"),
    ("alltoall", 128, 1525, "f8", 1, "move-alltoall"), ("alltoall", 31, 60001, "i4", 1, "move-alltoall"),
    ("alltoall", 7, 2500001, "u1", 1, "move-alltoall"), ("alltoall", 128, 20, "f8", 0, "copy"),
    ("allreduce", 5, 1000, "f8", 0, "gather"), ("allreduce", 512, 20001, "f8", 1, "passes"),
    ("allreduce", 300, 160003, "f8", 1, "rows-many"), ("allreduce", 512, 20001, "f4", 1, "passes"),
    ("bcast", 200, 4097, "u1", 0, "gather"), ("bcast", 128, 2400001, "u1", 0, "move-fan"),
    ("bcast", 256, 957025, "u1", 0, "move-fan"), ("bcast", 512, 51268, "f8", 0, "move-fan"),
    ("reduce", 3, 1025, "u1", 0, "gather"), ("reduce", 128, 600001, "i2", 0, "gather"),
    ("alltoall", 256, 257, "u1", 1, "move-alltoall"), ("alltoall", 256, 256, "u1", 1, "copy"),
    ("alltoall", 730, 145, "u1", 1, "move-alltoall"), ("alltoall", 256, 255, "i2", 1, "copy"),
]


@pytest.mark.parametrize("call,ranks,count,dt,skew,form", FORMS)
def test_the_form_of_a_call(cover, call, ranks, count, dt, skew, form):
    t = TYPES[dt]
    r = subprocess.run([cover, "one", str(OPS[call]), str(ranks), str(count), str(t[0]), str(t[1]), str(skew)],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:]
    assert form in r.stdout.split("forms ")[1].split(), r.stdout


@pytest.mark.parametrize("call,ranks,count,skew", [("bcast", 64, 1000000, 0), ("bcast", 64, 1000001, 1),
                                                   ("allgather", 24, 70000, 0), ("allgather", 24, 70001, 1)])
def test_the_form_of_a_call_among_others(cover, call, ranks, count, skew):
    r = subprocess.run([cover, "one", str(OPS[call]), str(ranks), str(count), "13", "8", str(skew), "3", "1.157e9"],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:]
    assert "move-fan" in r.stdout.split("forms ")[1].split(), r.stdout
