"""Folds over more ranks than a block keeps addresses for beside its ring.

Sizes around the lines of the choice of tiles (a gather tile that fills a warp
or not, rows for each SM, vectors streamed) and of the rank counts that its
tables distinguish, aligned and with odd buffers, against a fold on the device
in rank order: every byte equal, and the bytes around the buffers untouched.
"""
import importlib.util
import os
import sys

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api(gpu_built):
    spec = importlib.util.spec_from_file_location("gpumpi_coll", os.path.join(gpu_built.PKG, "gpumpi_coll.py"))
    mod = importlib.util.module_from_spec(spec)
    sys.modules[spec.name] = mod
    spec.loader.exec_module(mod)
    return mod, mod.bind(gpu_built.load_library())


def _check(api, p, n, dt, op, batched):
    import torch

    coll, lib = api
    es = torch.empty(0, dtype=getattr(torch, dt)).element_size()
    g = torch.Generator(device="cuda").manual_seed(p * 31 + n)
    shape = (p, n)
    if dt.startswith("float"):
        x = torch.rand(shape, dtype=getattr(torch, dt), device="cuda", generator=g) * 2 - 1
    else:
        x = torch.randint(0 if dt == "uint8" else -(1 << 20), 256 if dt == "uint8" else 1 << 20, shape, device="cuda", generator=g).to(getattr(torch, dt))
    acc = x[0].clone()
    for q in range(1, p):
        acc = x[q] + acc if op == "sum" else torch.maximum(x[q], acc)
    guard = 32
    out = torch.full((p * n + 2 * guard,), 77, dtype=x.dtype, device="cuda")
    red = torch.full((n + 2 * guard,), 77, dtype=x.dtype, device="cuda")
    comm = coll.Comm(lib, p)
    keep = []
    sends = [x.data_ptr() + r * n * es for r in range(p)]
    recvs = [out.data_ptr() + (guard + r * n) * es for r in range(p)]
    code = {"sum": coll.OP_SUM, "max": coll.OP_MAX}[op]
    # the root's buffer is the only one of the Reduce that is used
    plan = coll.Plan(lib, [
        coll.make_desc(comm, coll.COLL_ALLREDUCE, dt, n, sends, recvs, code, 0, keep),
        coll.make_desc(comm, coll.COLL_REDUCE, dt, n, sends, [red.data_ptr() + guard * es] * p, code, p - 1, keep),
    ], threads=64, batched=batched)
    plan.launch()
    torch.cuda.synchronize()
    assert coll.status(lib) is None
    plan.close()
    comm.close()
    assert torch.equal(out[guard:-guard].view(p, n), acc.expand(p, n))
    assert torch.equal(red[guard:-guard], acc)
    for t in (out, red):
        assert (t[:guard] == 77).all() and (t[-guard:] == 77).all()


@pytest.mark.parametrize("batched", [False, True])
@pytest.mark.parametrize("p", [256, 257, 300, 512, 513, 768, 769, 1024, 2048])
@pytest.mark.parametrize("n", [1, 31, 33, 500, 2000, 6001, 20000, 20001])
def test_folds_of_many_ranks(api, p, n, batched):
    _check(api, p, n, "float64", "sum", batched)
    _check(api, p, n, "int32", "max", batched)


@pytest.mark.parametrize("p,n,dt", [(257, 160002, "float64"), (257, 160003, "float64"), (384, 330000, "float32"),
                                    (768, 165000, "float64"), (769, 165000, "float64"), (1024, 60000, "float64"),
                                    (1024, 60001, "float64"), (2048, 60000, "float64"), (2048, 130001, "int32"),
                                    (640, 700000, "uint8"), (640, 700001, "uint8")])
@pytest.mark.parametrize("batched", [False, True])
def test_long_folds_of_many_ranks(api, p, n, dt, batched):
    _check(api, p, n, dt, "max" if dt == "uint8" else "sum", batched)
