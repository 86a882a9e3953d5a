"""Launch-ordered plans in spread form against the rank form and the host.

A launch-ordered plan whose calls leave the schedule to the runtime runs as
independent tiles over the whole GPU; with flag rounds (set_sync(1)) the same
plan runs one block per rank.  Both are exact, so every output byte must be
equal, and the bytes around each output untouched; Allreduce is also compared
with a host fold in rank order (acc = x_0; acc = op(x_q, acc)).
"""
import ctypes
import importlib.util
import os
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# element types of the API: datatype value, NumPy type
TYPES = {"i1": (6, np.int8), "u1": (29, np.uint8), "i2": (1, np.int16), "u2": (8, np.uint16), "i4": (2, np.int32),
         "u4": (9, np.uint32), "i8": (20, np.int64), "u8": (11, np.uint64), "f4": (12, np.float32),
         "f8": (13, np.float64)}
OPS = {"max": 0, "min": 1, "sum": 2, "prod": 3}


@pytest.fixture(scope="module")
def api(gpu_built):
    spec = importlib.util.spec_from_file_location("gpumpi_coll", os.path.join(gpu_built.PKG, "gpumpi_coll.py"))
    mod = importlib.util.module_from_spec(spec)
    sys.modules[spec.name] = mod
    spec.loader.exec_module(mod)
    return mod, mod.bind(gpu_built.load_library())


def _values(rng, count, dt):
    t = TYPES[dt][1]
    if dt in ("f4", "f8"):
        return rng.uniform(-1.5, 1.5, count).astype(t)
    info = np.iinfo(t)
    return rng.integers(info.min, info.max, count, dtype=t, endpoint=True)


def _fold(xs, op):
    acc = xs[0].copy()
    with np.errstate(over="ignore", under="ignore"):
        for x in xs[1:]:
            acc = {"sum": lambda: x + acc, "prod": lambda: x * acc, "max": lambda: np.where(x > acc, x, acc),
                   "min": lambda: np.where(x > acc, acc, x)}[op]()
    return acc


class Buffers:
    """P buffers of `count` elements in one allocation, 64 guard bytes around each, starting `skew` elements
    (times the rank) past a 16-byte boundary."""

    def __init__(self, torch, p, count, dt, skew, values=None):
        es = np.dtype(TYPES[dt][1]).itemsize
        self.stride = (count * es + 15) // 16 * 16 + 160
        self.host = np.full(p * self.stride, 0xA5, dtype=np.uint8)
        self.at = [r * self.stride + 64 + (r * skew * es) % 16 for r in range(p)]
        self.n = count * es
        if values is not None:
            for a, v in zip(self.at, values):
                self.host[a:a + self.n] = v.view(np.uint8)
        self.dev = torch.from_numpy(self.host.copy()).cuda()
        self.ptrs = [self.dev.data_ptr() + a for a in self.at]

    def reset(self, torch):
        self.dev.copy_(torch.from_numpy(self.host))

    def rows(self, dt):
        """The buffers' contents; everything outside them must be as it was."""
        now = self.dev.cpu().numpy()
        inside = np.zeros(len(now), dtype=bool)
        for a in self.at:
            inside[a:a + self.n] = True
        assert np.array_equal(now[~inside], self.host[~inside]), "bytes outside the buffers changed"
        return [now[a:a + self.n].copy().view(TYPES[dt][1]) for a in self.at]


def _run(api, p, n, dt, op, skew, batched, named=False):
    import torch

    coll, lib = api
    rng = np.random.default_rng(p * 100003 + n * 7 + skew)
    comm = coll.Comm(lib, p)
    keep, descs, outs = [], [], []

    def call(kind, count, send, recv, root=0):
        s = coll.ptr_array(send.ptrs) if send else None
        r = coll.ptr_array(recv.ptrs)
        keep.extend([s, r, send, recv])
        d = coll.Desc(comm.h, kind, TYPES[dt][0], OPS[op], root, count,
                      ctypes.cast(s, ctypes.POINTER(ctypes.c_void_p)) if send else None,
                      ctypes.cast(r, ctypes.POINTER(ctypes.c_void_p)), 0, 0)
        descs.append(d)
        outs.append(recv)

    xs = [_values(rng, n, dt) for _ in range(p)]
    call(coll.COLL_ALLREDUCE, n, Buffers(torch, p, n, dt, skew, xs), Buffers(torch, p, n, dt, skew))
    place = Buffers(torch, p, n, dt, skew, xs)
    call(coll.COLL_ALLREDUCE, n, place, place)
    call(coll.COLL_REDUCE, n, Buffers(torch, p, n, dt, skew, xs), Buffers(torch, p, n, dt, 0), p - 1)
    call(coll.COLL_BCAST, n, None, Buffers(torch, p, n, dt, skew, [_values(rng, n, dt) for _ in range(p)]), p // 2)
    per = max(1, n // p)
    call(coll.COLL_ALLTOALL, per, Buffers(torch, p, per * p, dt, skew, [_values(rng, per * p, dt) for _ in range(p)]),
         Buffers(torch, p, per * p, dt, 3 * skew))
    call(coll.COLL_ALLGATHER, per, Buffers(torch, p, per, dt, skew, [_values(rng, per, dt) for _ in range(p)]),
         Buffers(torch, p, per * p, dt, 5 * skew))
    for d in descs if named else []:
        d.algo = {coll.COLL_BCAST: 1, coll.COLL_REDUCE: 2, coll.COLL_ALLREDUCE: 3}.get(d.op, 4)
    plan = coll.Plan(lib, descs, threads=64, batched=batched)
    assert plan.launch_ordered
    got = []
    for mode in (0, 1):
        plan.set_sync(mode)
        for o in outs:
            o.reset(torch)
        torch.cuda.synchronize()
        plan.launch()
        torch.cuda.synchronize()
        assert coll.status(lib) is None
        got.append([o.rows(dt) for o in outs])
    plan.close()
    comm.close()
    for k, (a, b) in enumerate(zip(*got)):
        if k == 1:
            continue   # in place: with flag rounds a rank may fold a buffer that its owner has written already
        for r in range(p):
            assert a[r].tobytes() == b[r].tobytes(), "call %d rank %d" % (k, r)
    want = _fold(xs, op)
    for r in range(p):
        assert got[0][0][r].tobytes() == want.tobytes() and got[0][1][r].tobytes() == want.tobytes()
    assert got[0][2][p - 1].tobytes() == want.tobytes()


@pytest.mark.parametrize("dt", sorted(TYPES))
@pytest.mark.parametrize("op", ["max", "min", "sum", "prod"])
def test_every_type_and_operator(api, dt, op):
    _run(api, 5, 1000, dt, op, 0, True)
    _run(api, 9, 333, dt, op, 1, False)


@pytest.mark.parametrize("p,n", [(1, 1), (2, 1), (3, 31), (33, 32), (64, 255), (257, 1), (257, 300)])
@pytest.mark.parametrize("dt", ["f8", "i4"])
@pytest.mark.parametrize("skew", [0, 1])
def test_short_calls(api, p, n, dt, skew):
    _run(api, p, n, dt, "sum", skew, True)


@pytest.mark.parametrize("p,n", [(2, 4096), (3, 50001), (8, 131072), (8, 262149), (48, 65537), (300, 6001)])
@pytest.mark.parametrize("dt,skew", [("f8", 0), ("f8", 1), ("i4", 0), ("i4", 1), ("u1", 0), ("u1", 1), ("u2", 3)])
def test_long_calls(api, p, n, dt, skew):
    _run(api, p, n, dt, "max" if dt in ("u1", "u2") else "sum", skew, True)


@pytest.mark.parametrize("batched", [True, False])
@pytest.mark.parametrize("per", [95, 96, 128, 129, 171, 512, 513, 2047, 2500])
@pytest.mark.parametrize("dt", ["i4", "f8"])
def test_blocks_around_whole_chunks(api, per, dt, batched):
    """Alltoall and Allgather blocks of 4- and 8-byte units that fill a warp's
    chunks exactly, just miss them, or are too ragged for them."""
    _run(api, 5, 5 * per, dt, "sum", 1, batched)


@pytest.mark.parametrize("batched", [True, False])
@pytest.mark.parametrize("p,n,skew", [(3, 31, 1), (16, 20000, 0), (8, 262149, 1)])
def test_calls_that_name_the_schedule_of_the_tiles(api, p, n, skew, batched):
    _run(api, p, n, "f8", "sum", skew, batched, named=True)
    _run(api, p, n, "u2", "max", skew, batched, named=True)


@pytest.mark.parametrize("p,n,skew", [(2, 64, 0), (7, 1001, 1), (48, 20000, 0), (257, 999, 1), (64, 65537, 0)])
def test_dependent_calls_in_levels(api, p, n, skew):
    """Calls that use each other's results, write buffers that earlier calls
    read, and one that depends on nothing, in one launch: the same bytes as
    with flag rounds, launch after launch."""
    import torch

    coll, lib = api
    rng = np.random.default_rng(p + n)
    comm, other = coll.Comm(lib, p), coll.Comm(lib, 3)
    per = n // p
    x, w, s = (Buffers(torch, p, n, "f8", skew, [_values(rng, n, "f8") for _ in range(p)]) for _ in range(3))
    j = Buffers(torch, p, per * p, "f8", skew)
    y, z = (Buffers(torch, 3, 100, "i4", skew, [_values(rng, 100, "i4") for _ in range(3)]) for _ in range(2))
    keep = []

    def call(c, kind, dt, count, send, recv, op=2, root=0):
        return coll.make_desc(c, kind, {"f8": "float64", "i4": "int32"}[dt], count, send.ptrs if send else None,
                              recv.ptrs, op, root, keep)

    plan = coll.Plan(lib, [
        call(comm, coll.COLL_ALLREDUCE, "f8", n, x, w),              # w: the sum
        call(comm, coll.COLL_ALLTOALL, "f8", per, w, s),             # reads w
        call(other, coll.COLL_ALLREDUCE, "i4", 100, y, z),           # on its own
        call(comm, coll.COLL_ALLGATHER, "f8", per, s, j),            # reads s
        call(comm, coll.COLL_REDUCE, "f8", per * p, j, x, 0, p - 1),  # writes what the first call read
        call(comm, coll.COLL_BCAST, "f8", per * p, None, x, 0, p - 1),
        call(comm, coll.COLL_ALLREDUCE, "f8", per * p, x, w, 3),     # writes w again
    ], threads=64, batched=True)
    assert not plan.launch_ordered
    outs = [x, w, s, j, y, z]
    types = ["f8"] * 4 + ["i4"] * 2
    got = []
    for mode in (0, 0, 1):
        plan.set_sync(mode)
        if len(got) == 1:
            plan.capture()
        for o in outs:
            o.reset(torch)
        torch.cuda.synchronize()
        plan.launch()
        torch.cuda.synchronize()
        assert coll.status(lib) is None
        got.append([o.rows(t) for o, t in zip(outs, types)])
    plan.close()
    comm.close()
    other.close()
    for a, b, c in zip(*got):
        for u, v, t in zip(a, b, c):
            assert u.tobytes() == v.tobytes() == t.tobytes()


@pytest.mark.parametrize("batched", [True, False])
def test_launches_of_a_stream_keep_their_order(api, batched):
    """Launches overlap the end of the one before, but read nothing it writes
    too early: long and short plans, copies and kernels of one stream in turn,
    directly and recorded into a graph, each using the one before."""
    import torch

    coll, lib = api
    p, n = 6, 100000
    g = torch.Generator().manual_seed(3)
    x = torch.randint(-1000, 1000, (p, n), dtype=torch.int32, generator=g).cuda()
    a, b, c = (torch.zeros(p, n, dtype=torch.int32, device="cuda") for _ in range(3))
    comm = coll.Comm(lib, p)
    keep = []
    rows = lambda t, k=p: [t.data_ptr() + r * n * 4 for r in range(k)]  # noqa: E731
    add = coll.Plan(lib, [coll.make_desc(comm, coll.COLL_ALLREDUCE, "int32", n, rows(a), rows(b), 2, 0, keep)],
                    threads=64, batched=batched)
    spread = coll.Plan(lib, [coll.make_desc(comm, coll.COLL_BCAST, "int32", 5, None, rows(b), 0, 1, keep)],
                       threads=64, batched=batched)
    empty = coll.Plan(lib, [coll.make_desc(comm, coll.COLL_ALLREDUCE, "int32", 0, rows(a), rows(b), 2, 0, keep)],
                      threads=64, batched=batched)
    turn = coll.Plan(lib, [coll.make_desc(comm, coll.COLL_ALLTOALL, "int32", n // p, rows(b), rows(c), 0, 0, keep)],
                     threads=64, batched=batched)

    def steps(stream):
        a.copy_(x)                            # a copy, then plans, then kernels, over and over
        for k in range(4):
            add.launch(stream)                # b = sum of a
            spread.launch(stream)             # a short one that writes b
            empty.launch(stream)
            turn.launch(stream)               # c from b
            torch.add(c, k, out=a)            # a from c
            c.zero_()

    want = x.cpu().numpy()
    per = n // p
    with np.errstate(over="ignore"):
        for k in range(4):
            s = np.tile(want.sum(0, dtype=np.int32), (p, 1))
            out = np.zeros_like(s)
            for r in range(p):
                for q in range(p):
                    out[r, q * per:(q + 1) * per] = s[q, r * per:(r + 1) * per]
            want = out + np.int32(k)
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        steps(st.cuda_stream)
    torch.cuda.synchronize()
    assert np.array_equal(a.cpu().numpy(), want)
    steps(0)
    torch.cuda.synchronize()
    assert np.array_equal(a.cpu().numpy(), want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        steps(st.cuda_stream)
    for _ in range(3):
        a.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(a.cpu().numpy(), want)
    for plan in (add, spread, empty, turn):
        plan.close()
    comm.close()


@pytest.mark.parametrize("p,n", [(1, 1), (2, 5), (31, 4097), (256, 1), (256, 40001)])
@pytest.mark.parametrize("dt,skew", [("f8", 0), ("f8", 1), ("i4", 1), ("u2", 1)])
def test_noalloc_allreduce_matches_the_host(api, p, n, dt, skew):
    import torch

    coll, lib = api
    lib.gpumpi_allreduce_noalloc.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.POINTER(ctypes.c_void_p),
                                             ctypes.c_int, ctypes.c_uint64, ctypes.c_int, ctypes.c_int, ctypes.c_int,
                                             ctypes.c_void_p]
    rng = np.random.default_rng(p * 17 + n)
    xs = [_values(rng, n, dt) for _ in range(p)]
    send, recv = Buffers(torch, p, n, dt, skew, xs), Buffers(torch, p, n, dt, 3 * skew)
    for _ in range(2):
        recv.reset(torch)
        rc = lib.gpumpi_allreduce_noalloc(coll.ptr_array(send.ptrs), coll.ptr_array(recv.ptrs), p, n, TYPES[dt][0],
                                          OPS["sum"], 128, None)
        assert rc == 0, lib.gpumpi_last_error().decode()
        want = _fold(xs, "sum")
        assert all(row.tobytes() == want.tobytes() for row in recv.rows(dt))


@pytest.mark.parametrize("how", ["pinned", "in place", "shared input", "pageable", "captured"])
def test_host_buffer_calls_in_groups(api, how):
    """A host-buffer call large enough to copy in, run and copy out in groups
    gives the bytes that the one-after-another form (flag rounds) gives, call
    after call with new inputs; also where the groups do not apply: results over
    the inputs in host memory, two calls filling one device buffer, pageable
    memory, a stream under capture."""
    import torch

    coll, lib = api
    rng = np.random.default_rng(17)
    shapes = [("allreduce", 16, 20000), ("alltoall", 16, 1300), ("bcast", 16, 20001), ("reduce", 5, 40000),
              ("allgather", 5, 7001), ("allreduce", 5, 30001)]
    comms = {p: coll.Comm(lib, p) for p in (16, 5)}
    kinds = {"allreduce": coll.COLL_ALLREDUCE, "alltoall": coll.COLL_ALLTOALL, "bcast": coll.COLL_BCAST,
             "reduce": coll.COLL_REDUCE, "allgather": coll.COLL_ALLGATHER}
    keep, descs, hs, hr, ins, outs = [], [], [], [], [], []
    first = None
    for kind, p, n in shapes:
        ns = n * p if kind == "alltoall" else n
        nr = n * p if kind in ("alltoall", "allgather") else n
        dev_in = torch.zeros(p, ns, dtype=torch.float64, device="cuda")
        if how == "shared input" and kind == "allreduce" and p == 5:
            dev_in = first            # the Reduce's input, filled twice by one call
        elif kind == "reduce":
            first = dev_in
        dev_out = torch.zeros(p, nr, dtype=torch.float64, device="cuda")
        host_in = torch.from_numpy(rng.uniform(-1, 1, (p, dev_in.shape[1])))
        host_out = torch.zeros(p, nr, dtype=torch.float64)
        if how != "pageable":
            host_in, host_out = host_in.pin_memory(), host_out.pin_memory()
        if how == "in place" and ns == nr and kind != "bcast":
            host_out = host_in
        keep += [dev_in, dev_out]
        rows = lambda t, k=p: [t.data_ptr() + r * t.shape[1] * 8 for r in range(k)]  # noqa: E731
        descs.append(coll.make_desc(comms[p], kinds[kind], "float64", n, None if kind == "bcast" else rows(dev_in),
                                    rows(dev_out), coll.OP_SUM, p - 1 if kind in ("reduce", "bcast") else 0, keep))
        hs += rows(host_in)
        hr += rows(host_out)
        ins.append(host_in)
        outs.append(host_out)
    plan = coll.Plan(lib, descs, threads=64, batched=True)
    st = torch.cuda.Stream()
    got = []
    for mode in (0, 1):
        plan.set_sync(mode)
        rng = np.random.default_rng(23)
        res = []
        for _ in range(3):
            for t in ins:
                t.copy_(torch.from_numpy(rng.uniform(-1, 1, tuple(t.shape))))
            for t, i in zip(outs, ins):
                if t is not i:
                    t.fill_(-3.0)
            if how == "captured" and mode == 0:
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=st):
                    plan.run_host(hs, hr, st.cuda_stream)
                graph.replay()
            else:
                bi, bo = plan.run_host(hs, hr, st.cuda_stream)
                assert bi + bo > 4 << 20
            torch.cuda.synchronize()
            assert coll.status(lib) is None
            res.append([t.numpy().copy() for t in outs])
        got.append(res)
    plan.close()
    for c in comms.values():
        c.close()
    for a, b in zip(*got):
        for x, y in zip(a, b):
            assert x.tobytes() == y.tobytes()


@pytest.mark.parametrize("n", [17, 60001, 262144])
def test_plain_launches_without_a_common_buffer_overlap(api, n):
    """A plain plan's launches wait for one another only where they share
    memory; they still see what the stream ran before the plan, and what follows
    the plan sees all of them.  Inputs change and outputs are cleared between
    the launches, directly and recorded into a graph."""
    import torch

    coll, lib = api
    p, q, m, rounds = 6, 3, 500, 6
    g = torch.Generator().manual_seed(n)
    n = n // p * p
    a0 = torch.randint(-1000, 1000, (p, n), dtype=torch.int32, generator=g)
    d0 = torch.randint(-1000, 1000, (q, m), dtype=torch.int32, generator=g)
    a, d = torch.zeros_like(a0, device="cuda"), torch.zeros_like(d0, device="cuda")
    b, c, h = (torch.zeros(p, n, dtype=torch.int32, device="cuda") for _ in range(3))
    e = torch.zeros(q, m, dtype=torch.int32, device="cuda")
    f = torch.zeros(q, q * m, dtype=torch.int32, device="cuda")
    w = torch.zeros(p, n, dtype=torch.int32, device="cuda")
    big, small = coll.Comm(lib, p), coll.Comm(lib, q)
    keep = []
    rows = lambda t: [t.data_ptr() + r * t.shape[1] * 4 for r in range(t.shape[0])]  # noqa: E731
    plan = coll.Plan(lib, [
        coll.make_desc(big, coll.COLL_ALLREDUCE, "int32", n, rows(a), rows(b), 2, 0, keep),
        coll.make_desc(big, coll.COLL_ALLTOALL, "int32", n // p, rows(a), rows(c), 0, 0, keep),
        coll.make_desc(big, coll.COLL_REDUCE, "int32", n, rows(a), rows(h), 0, 2, keep),
        coll.make_desc(big, coll.COLL_BCAST, "int32", n, None, rows(w), 0, 1, keep),
        coll.make_desc(small, coll.COLL_ALLREDUCE, "int32", m, rows(d), rows(e), 2, 0, keep),
        coll.make_desc(small, coll.COLL_ALLGATHER, "int32", m, rows(e), rows(f), 0, 0, keep),   # uses the one before
        coll.make_desc(big, coll.COLL_ALLREDUCE, "int32", n, rows(w), rows(c), 2, 0, keep),     # and these two
        coll.make_desc(big, coll.COLL_ALLREDUCE, "int32", n, rows(h), rows(w), 1, 0, keep),
    ], threads=64, batched=False)
    outs = [b, c, h, w, e, f]
    sums = [torch.zeros_like(t) for t in outs]

    def steps(stream):
        a.copy_(a0_dev)
        d.copy_(d0_dev)
        for s in sums:
            s.zero_()
        for k in range(rounds):
            a.add_(k)
            d.add_(k)
            w.copy_(a)
            plan.launch(stream)
            for s, t in zip(sums, outs):
                s.add_(t)
                t.zero_()

    a0_dev, d0_dev = a0.cuda(), d0.cuda()
    want = [np.zeros(t.shape, dtype=np.int32) for t in outs]
    x, y = a0.numpy().copy(), d0.numpy().copy()
    for k in range(rounds):
        x, y = x + np.int32(k), y + np.int32(k)
        hh = np.zeros((p, n), dtype=np.int32)
        hh[2] = x.max(0)
        ee = np.tile(y.sum(0, dtype=np.int32), (q, 1))
        got = [np.tile(x.sum(0, dtype=np.int32), (p, 1)), np.tile(x[1] * np.int32(p), (p, 1)), hh,
               np.tile(hh.min(0), (p, 1)), ee, np.tile(ee.reshape(-1), (q, 1))]
        for u, v in zip(want, got):
            u += v
    st = torch.cuda.Stream()
    torch.cuda.synchronize()

    def check():
        torch.cuda.synchronize()
        assert coll.status(lib) is None
        for s, u in zip(sums, want):
            assert np.array_equal(s.cpu().numpy(), u)

    for _ in range(3):
        with torch.cuda.stream(st):
            steps(st.cuda_stream)
        check()
    plan.capture()
    with torch.cuda.stream(st):
        steps(st.cuda_stream)
    check()
    plan.set_sync(0)   # drops the plan's own graph
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        steps(st.cuda_stream)
    for _ in range(3):
        graph.replay()
        check()
    plan.close()
    big.close()
    small.close()


def test_two_threads_on_one_stream_take_turns(api):
    """Plain plans of two threads on one stream: each plan's launches stay
    together, so a launch that does not wait for its own plan's earlier ones
    still waits for the other thread's.  Each plan writes the buffer that the
    other one's later launches read; every result must be one plan's or the
    other's, whole."""
    import threading

    import torch

    coll, lib = api
    p, n, rounds = 4, 200000, 150
    comm = coll.Comm(lib, p)
    keep = []
    rows = lambda t: [t.data_ptr() + r * n * 4 for r in range(p)]  # noqa: E731
    shared = torch.full((p, n), 3, dtype=torch.int32, device="cuda")
    ins = [torch.full((p, n), v, dtype=torch.int32, device="cuda") for v in (1, 2)]
    outs = [[torch.zeros(p, n, dtype=torch.int32, device="cuda") for _ in range(2)] for _ in range(2)]
    plans = []
    for x, (a, b) in zip(ins, outs):
        plans.append(coll.Plan(lib, [
            coll.make_desc(comm, coll.COLL_ALLREDUCE, "int32", n, rows(x), rows(a), 2, 0, keep),
            coll.make_desc(comm, coll.COLL_ALLREDUCE, "int32", n, rows(shared), rows(b), 2, 0, keep),
            coll.make_desc(comm, coll.COLL_ALLREDUCE, "int32", n, rows(x), rows(shared), 2, 0, keep),
        ], threads=64, batched=False))
    st = torch.cuda.Stream()
    torch.cuda.synchronize()

    def work(k):
        with torch.cuda.stream(st):
            for _ in range(rounds):
                plans[k].launch(st.cuda_stream)

    for _ in range(3):
        threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        torch.cuda.synchronize()
        assert coll.status(lib) is None
        for k in range(2):
            assert (outs[k][0] == p * (k + 1)).all()
            b = outs[k][1].cpu().numpy()
            assert (b == b[0, 0]).all() and b[0, 0] in (3 * p, p * p, 2 * p * p)
        s = shared.cpu().numpy()
        assert (s == s[0, 0]).all() and s[0, 0] in (p, 2 * p)
    for plan in plans:
        plan.close()
    comm.close()
