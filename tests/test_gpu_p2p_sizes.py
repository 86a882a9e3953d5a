"""Blocking point-to-point messages at the edges of the leader's copy paths."""
import pytest

from conftest import run_oracle

from kat_cases import check_all_ok

GPU_OPTS = ["--timeout-ms", "20000", "--max-seconds", "120"]


def test_sizes_on_the_host(oracle_built):
    check_all_ok(run_oracle("kat_p2p", ["sizes"], nranks=2, timeout=120), "sizes", 2)


@pytest.mark.gpu
@pytest.mark.parametrize("extra", [[], ["--one-cluster"]], ids=["grid", "one-cluster"])
def test_gpu_sizes(gpu_built, extra):
    res = gpu_built.run_program("kat_p2p", ["sizes"], nranks=2, extra=GPU_OPTS + extra, timeout=180)
    check_all_ok(res, "sizes", 2)
