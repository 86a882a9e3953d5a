"""Forms of tiles that it takes a large call to reach, and values that a fold must not change.

Each call runs as tiles and is compared, byte for byte, with the same fold or
copy by PyTorch on the device; the bytes around every buffer stay untouched.
tests/test_spread_cover.py checks on the CPU that these sizes reach the form
they are meant for.
"""
import importlib.util
import os
import sys

import pytest

pytestmark = pytest.mark.gpu

GUARD = 64   # bytes around each buffer


@pytest.fixture(scope="module")
def api(gpu_built):
    spec = importlib.util.spec_from_file_location("gpumpi_coll", os.path.join(gpu_built.PKG, "gpumpi_coll.py"))
    mod = importlib.util.module_from_spec(spec)
    sys.modules[spec.name] = mod
    spec.loader.exec_module(mod)
    return mod, mod.bind(gpu_built.load_library())


class Rows:
    """P buffers of n elements in one allocation, buffer r starting r * skew elements past a 16-byte boundary."""

    def __init__(self, p, n, dt, skew, seed=None):
        import torch

        self.dt = getattr(torch, dt)
        es = torch.empty(0, dtype=self.dt).element_size()
        self.bytes = n * es
        step = (self.bytes + 15) // 16 * 16 + 2 * GUARD + 16
        self.mem = torch.empty(p * step, dtype=torch.uint8, device="cuda")
        self.mem.fill_(0xA5)
        self.at = [r * step + GUARD + r * skew * es % 16 for r in range(p)]
        if seed is not None:
            g = torch.Generator(device="cuda").manual_seed(seed)
            for r in range(p):
                row = self.row(r)
                if dt.startswith("float"):
                    row.uniform_(-1.5, 1.5, generator=g)
                else:
                    row.random_(0, 200, generator=g)
        self.ptrs = [self.mem.data_ptr() + a for a in self.at]

    def row(self, r):
        m = self.mem[self.at[r]:self.at[r] + self.bytes]
        if m.data_ptr() % m.new_empty(0, dtype=self.dt).element_size():
            raise AssertionError("alignment")
        return _typed(m, self.dt)

    def outside_untouched(self):
        end = 0
        for a in self.at + [len(self.mem)]:
            assert (self.mem[end:a] == 0xA5).all(), "bytes around the buffers changed"
            end = a + self.bytes


def _typed(m, dt):
    """Bytes as elements of dt; the storage offset is a multiple of the element's size."""
    import torch

    if dt == torch.uint8:
        return m
    es = torch.empty(0, dtype=dt).element_size()
    whole = torch.empty(0, dtype=dt, device="cuda").set_(m.untyped_storage(), m.storage_offset() // es, (len(m) // es,))
    assert whole.data_ptr() == m.data_ptr()
    return whole


def _same(a, b):
    import torch

    return torch.equal(a.contiguous().view(torch.uint8), b.contiguous().view(torch.uint8))


def _fold(xs, p, op):
    import torch

    acc = xs(0).clone()
    for q in range(1, p):
        x = xs(q)
        acc = {"sum": lambda: x + acc, "max": lambda: torch.where(x > acc, x, acc),
               "min": lambda: torch.where(x > acc, acc, x)}[op]()
    return acc


def _launch(api, descs, batched):
    import torch

    coll, lib = api
    plan = coll.Plan(lib, descs, threads=64, batched=batched)
    plan.launch()
    torch.cuda.synchronize()
    assert coll.status(lib) is None
    plan.close()


class Call:
    def __init__(self, api, kind, p, n, dt, skew, op="sum", values=None):
        coll, lib = api
        self.kind, self.p, self.n, self.op, self.root = kind, p, n, op, p // 2
        self.keep = []
        self.comm = coll.Comm(lib, p)
        ns = n * p if kind == "alltoall" else n
        nr = n * p if kind in ("alltoall", "allgather") else n
        self.send = Rows(p, ns, dt, skew, seed=p + n) if kind != "bcast" else None
        # of a Reduce only the root's buffer is used
        self.recv = Rows(p if kind != "reduce" else 1, nr, dt, 3 * skew, seed=n if kind == "bcast" else None)
        if values is not None:
            values(self.send)
        if kind == "bcast":
            self.want = self.recv.row(self.root).clone()
        code = {"bcast": coll.COLL_BCAST, "reduce": coll.COLL_REDUCE, "allreduce": coll.COLL_ALLREDUCE,
                "alltoall": coll.COLL_ALLTOALL, "allgather": coll.COLL_ALLGATHER}[kind]
        red = {"sum": coll.OP_SUM, "max": coll.OP_MAX, "min": coll.OP_MIN}[op]
        self.desc = coll.make_desc(self.comm, code, dt, n, self.send.ptrs if self.send else None,
                                   self.recv.ptrs if kind != "reduce" else self.recv.ptrs * p, red, self.root, self.keep)

    def check(self):
        p, n = self.p, self.n
        if self.kind == "bcast":
            for r in range(p):
                assert _same(self.recv.row(r), self.want), "rank %d" % r
        elif self.kind in ("reduce", "allreduce"):
            want = _fold(self.send.row, p, self.op)
            for r in range(len(self.recv.at)):
                assert _same(self.recv.row(r), want), "rank %d" % r
        else:
            import torch

            sent = [self.send.row(q) for q in range(p)]
            for r in range(p):
                want = torch.cat([x[r * n:(r + 1) * n] for x in sent] if self.kind == "alltoall" else sent)
                assert _same(self.recv.row(r), want), "rank %d" % r
        self.recv.outside_untouched()
        if self.send:
            self.send.outside_untouched()
        self.comm.close()


# calls alone in their launch
ALONE = [
    # vectors streamed, and rows of odd buffers
    ("allreduce", 4, 1000000, "float64", 0), ("allreduce", 4, 1000001, "float64", 1), ("reduce", 64, 62497, "float64", 1),
    ("reduce", 64, 70001, "float64", 1), ("allreduce", 20, 600001, "int32", 1),
    # bulk copies to several destinations
    ("bcast", 16, 750000, "float64", 0), ("bcast", 16, 750001, "float64", 1), ("bcast", 16, 6000001, "uint8", 1),
    ("allgather", 100, 1000, "float64", 0), ("allgather", 100, 1001, "float64", 1), ("allgather", 100, 8001, "uint8", 1),
    # more than 250 MB
    ("reduce", 256, 126952, "float64", 0), ("reduce", 256, 126953, "float64", 1), ("reduce", 256, 1015624, "uint8", 0),
    ("allreduce", 160, 812500, "uint8", 0), ("allreduce", 256, 97656, "float64", 0), ("reduce", 320, 101560, "float64", 0),
    ("allreduce", 17, 2000001, "int32", 1), ("reduce", 512, 97657, "float64", 1),
    ("alltoall", 128, 1524, "float64", 0), ("alltoall", 31, 60000, "int32", 0), ("alltoall", 128, 1525, "float64", 1),
    ("alltoall", 31, 60001, "int32", 1), ("alltoall", 7, 2500001, "uint8", 1), ("alltoall", 128, 20, "float64", 0),
    # 1-byte types: whole vectors and a rest, pieces of half the length, short odd blocks
    ("bcast", 200, 4097, "uint8", 0), ("bcast", 128, 2400001, "uint8", 0), ("bcast", 256, 957025, "uint8", 0),
    ("bcast", 512, 51268, "float64", 0), ("reduce", 3, 1025, "uint8", 0), ("reduce", 128, 600001, "uint8", 0),
    ("allreduce", 256, 40001, "uint8", 0), ("allreduce", 64, 150001, "uint8", 0),
    ("alltoall", 256, 257, "uint8", 1), ("alltoall", 256, 256, "uint8", 1), ("alltoall", 730, 145, "uint8", 1),
]


@pytest.mark.parametrize("kind,p,n,dt,skew", ALONE)
def test_large_calls(api, kind, p, n, dt, skew):
    call = Call(api, kind, p, n, dt, skew, "max" if dt == "uint8" and "reduce" in kind else "sum")
    _launch(api, [call.desc], True)
    call.check()


@pytest.mark.parametrize("skew", [0, 1])
def test_bulk_copies_among_other_calls(api, skew):
    """A level of more than 1 GB, in which odd buffers go by bulk copies too."""
    calls = [Call(api, "bcast", 64, 1000000 + skew, "float64", skew), Call(api, "allgather", 24, 70000 + skew, "float64", skew),
             Call(api, "allreduce", 5, 33333, "int32", skew)]
    _launch(api, [c.desc for c in calls], True)
    for c in calls:
        c.check()


BEYOND = (1 << 32) + 12345


@pytest.mark.parametrize("kind,p,n,skew", [("bcast", 3, BEYOND, 1), ("bcast", 2, BEYOND // 16 * 16, 0),
                                           ("allreduce", 2, BEYOND, 1), ("allreduce", 2, BEYOND // 16 * 16, 0),
                                           ("alltoall", 2, BEYOND // 2, 1), ("alltoall", 2, BEYOND // 32 * 16, 0),
                                           ("allgather", 2, BEYOND // 2, 1)])
def test_buffers_beyond_4_gib(api, kind, p, n, skew):
    call = Call(api, kind, p, n, "uint8", skew, "max")
    _launch(api, [call.desc], False)
    call.check()


# gather tiles, vectors streamed, rows, passes over the sources, rows of many ranks
SPECIAL = [(5, 1000, 0), (4, 1000000, 0), (4, 1000001, 1), (512, 20001, 1), (300, 160003, 1)]


@pytest.mark.parametrize("p,n,skew", SPECIAL)
@pytest.mark.parametrize("op", ["max", "min", "sum"])
@pytest.mark.parametrize("dt", ["float64", "float32"])
def test_special_values_through_folds(api, p, n, skew, op, dt):
    """NaN, infinities, signed zeros and subnormals, in any order of ranks.  For
    MAX and MIN an operand stays or goes as `x > acc` says, and the kept one's
    bits are kept.  A NaN that is a sum has no sign of its own (rank blocks of
    two schedules differ in it): sums have theirs in the same places, and the
    same bits elsewhere."""
    import torch

    def values(rows):
        tiny = torch.finfo(getattr(torch, dt)).tiny / 4
        v = torch.tensor([float("nan"), float("inf"), -float("inf"), 0.0, -0.0, tiny, -tiny, 1.0, -1.0],
                         dtype=getattr(torch, dt), device="cuda")
        g = torch.Generator(device="cuda").manual_seed(n)
        for r in range(p):
            rows.row(r).copy_(v[torch.randint(0, len(v), (n,), device="cuda", generator=g)])

    call = Call(api, "allreduce", p, n, dt, skew, op, values)
    _launch(api, [call.desc], False)
    if op != "sum":
        call.check()
        return
    want = _fold(call.send.row, p, op)
    none = torch.isnan(want)
    for r in range(p):
        got = call.recv.row(r)
        assert torch.equal(torch.isnan(got), none) and _same(got[~none], want[~none]), "rank %d" % r
    call.recv.outside_untouched()
    call.comm.close()


def test_dependent_calls_with_another_schedule(api):
    """One call whose schedule tiles do not carry out keeps a plan of dependent
    calls in rank blocks, in one launch, with flag rounds between the calls."""
    import torch

    coll, lib = api
    p, n = 24, 5000
    comm, keep = coll.Comm(lib, p), []
    x, y, z = (Rows(p, n, "float64", 0, seed=s) for s in (1, None, None))
    descs = [coll.make_desc(comm, coll.COLL_ALLREDUCE, "float64", n, a.ptrs, b.ptrs, coll.OP_SUM, 0, keep, algo)
             for a, b, algo in ((x, y, 0), (y, z, 2))]
    plan = coll.Plan(lib, descs, threads=128, batched=True)
    assert not plan.launch_ordered
    before = lib.gpumpi_kernel_launches()
    plan.launch()
    torch.cuda.synchronize()
    assert coll.status(lib) is None
    assert lib.gpumpi_kernel_launches() == before + 1
    mid = _fold(x.row, p, "sum")
    out = _fold(lambda q: mid, p, "sum")
    for r in range(p):
        assert _same(y.row(r), mid) and _same(z.row(r), out)
    for t in (x, y, z):
        t.outside_untouched()
    plan.close()
    comm.close()
