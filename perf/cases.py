"""The work this runtime is measured on: collectives over device and host
buffers through the host API (include/gpumpi.h, dphpc-project_gb300/gpumpi_coll.py)
and a converted point-to-point program through its launcher.

Kinds of case:

  batch    16 communicators of 4..256 ranks (1024 ranks), each with Bcast,
           Allreduce(SUM) and Alltoall on int32 and FP64, n elements per rank,
           as one batched plan replayed as a CUDA graph: the benchmark's workload
  plain    one communicator, one launch per call: Bcast, Reduce, Allreduce,
           Alltoall and Allgather over five element types and three operators
  allreduce  one Allreduce of one communicator, one launch
  chain    a batched plan whose calls each use the one before: Allreduce,
           Alltoall of the sums, Allgather of a part, Reduce(MAX), Bcast: one
           step of an iterative solver, FP64
  host     three communicators from pinned host buffers and back
  noalloc  the allreduce for callers that may not allocate device memory
  p2p      a converted MPI program, message sizes 2^lg_min..2^lg_max bytes

Rank buffers of one call lie back to back in one allocation, as a [ranks, n]
tensor has them, so an odd n gives buffers that are aligned to their elements
only.
"""
import ctypes
import importlib.util
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SIZES = (4, 8, 12, 16, 24, 32, 40, 48, 56, 64, 72, 80, 88, 96, 128, 256)
HOST_SIZES = (128, 88, 40)   # one of the groups that the end-to-end benchmark splits SIZES into
TORCH = {"int32": torch.int32, "int64": torch.int64, "float32": torch.float32, "float64": torch.float64,
         "uint8": torch.uint8}
BYTES = {"int32": 4, "int64": 8, "float32": 4, "float64": 8, "uint8": 1}
THREADS = 128                # the default of the API and of the benchmark


def listed():
    return [
        # latency of a whole batch: every message is one element
        {"name": "batch_1", "kind": "batch", "n": 1},
        # short messages, odd length: rank buffers aligned to their elements only
        {"name": "batch_301", "kind": "batch", "n": 301},
        # middle sizes: 128 and 256 KiB per rank
        {"name": "batch_32768", "kind": "batch", "n": 32768},
        # middle sizes, odd length
        {"name": "batch_100003", "kind": "batch", "n": 100003},
        # the benchmark's headline size, about 61 GB of buffers
        {"name": "batch_1048576", "kind": "batch", "n": 1 << 20},
        # one launch per call, all collectives and most element types
        {"name": "plain_64r_50000", "kind": "plain", "ranks": 64, "n": 50000},
        # few ranks, long vectors: 16 MiB per rank
        {"name": "allreduce_8r_4Mi_f32", "kind": "allreduce", "ranks": 8, "n": 1 << 22, "dtype": "float32"},
        # the smallest call: one value per rank
        {"name": "allreduce_16r_1_f64", "kind": "allreduce", "ranks": 16, "n": 1, "dtype": "float64"},
        # calls that depend on each other, in one launch
        {"name": "chain_48r_20000", "kind": "chain", "ranks": 48, "n": 20000},
        # host buffers in, host buffers out
        {"name": "host_16384", "kind": "host", "n": 16384},
        # the call for fixed device-memory budgets, synchronous
        {"name": "noalloc_32r_4096", "kind": "noalloc", "ranks": 32, "n": 4096, "dtype": "float64"},
        # blocking messages of 8 B to 1 KiB between two ranks of a converted program
        {"name": "p2p_2r_8B_1KiB", "kind": "p2p", "ranks": 2, "lg_min": 3, "lg_max": 10, "iters": 12000},
    ]


def _log(rng, lo, hi):
    """An integer whose logarithm is uniform between those of lo and hi."""
    return int(min(hi, max(lo, round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["batch", "batch", "batch", "plain", "plain", "allreduce", "allreduce", "chain", "host",
                       "noalloc", "p2p"])
    if kind == "batch":
        return {"kind": kind, "n": _log(rng, 1, 1 << 20)}
    if kind == "plain":
        p = _log(rng, 2, 256)
        return {"kind": kind, "ranks": p, "n": _log(rng, 1, min(1 << 20, (1 << 23) // p))}
    if kind == "allreduce":
        p = _log(rng, 2, 128)
        return {"kind": kind, "ranks": p, "n": _log(rng, 1, (1 << 28) // p),
                "dtype": rng.choice(["float32", "float64", "int32", "int64"])}
    if kind == "chain":
        return {"kind": kind, "ranks": _log(rng, 4, 200), "n": _log(rng, 200, 1 << 17)}
    if kind == "host":
        return {"kind": kind, "n": _log(rng, 256, 1 << 15)}
    if kind == "noalloc":
        return {"kind": kind, "ranks": _log(rng, 2, 256), "n": _log(rng, 1, 1 << 17),
                "dtype": rng.choice(["float64", "int32"])}
    lg = rng.randint(3, 10)
    return {"kind": kind, "ranks": rng.choice([2, 2, 4, 8]), "lg_min": lg, "lg_max": lg + rng.randint(0, 2),
            "iters": _log(rng, 2000, 20000)}


# ------------------------------------------------------------------ inputs

def _calls(case):
    """The collective calls of a case: (kind, ranks, dtype, count, operator, root).
    Alltoall counts are elements per peer (at least 1)."""
    n = case["n"]
    if case["kind"] in ("batch", "host"):
        calls = []
        for p in SIZES if case["kind"] == "batch" else HOST_SIZES:
            for dt in ("int32", "float64"):
                calls += [("bcast", p, dt, n, "sum", 0), ("allreduce", p, dt, n, "sum", 0),
                          ("alltoall", p, dt, max(1, n // p), "sum", 0)]
        return calls
    p = case["ranks"]
    if case["kind"] == "plain":
        return [("bcast", p, "float64", n, "sum", p - 1), ("bcast", p, "uint8", n, "sum", 0),
                ("reduce", p, "float64", n, "sum", p // 2), ("reduce", p, "int64", n, "max", 0),
                ("allreduce", p, "float32", n, "sum", 0), ("allreduce", p, "int32", n, "min", 0),
                ("alltoall", p, "float32", max(1, n // p), "sum", 0),
                ("alltoall", p, "uint8", max(1, n // p), "sum", 0),
                ("allgather", p, "float64", max(1, n // p), "sum", 0),
                ("allgather", p, "int32", max(1, n // p), "sum", 0)]
    return [("allreduce", p, case["dtype"], n, "sum", 0)]


def _lengths(call):
    """Elements of a rank's send and receive buffers (Bcast works in place on the receive buffers)."""
    kind, p, _, n, _, _ = call
    if kind == "bcast":
        return 0, n
    if kind == "alltoall":
        return n * p, n * p
    if kind == "allgather":
        return n, n * p
    return n, n


def _layout(calls, side):
    """One flat tensor per (collective, type, position among its like): the
    offset of every call's buffers in it and its length in elements; calls start
    at 128-element steps."""
    at, total = [], {}
    for c in calls:
        key = (c[0], c[2])
        start = total.get(key, 0)
        at.append((key, start))
        total[key] = start + -(-(_lengths(c)[side] * c[1]) // 128) * 128
    return at, total


def _fill(t, dt, g):
    if dt == "uint8":
        t.random_(0, 256, generator=g)
    elif dt.startswith("int"):
        t.random_(-(1 << 20), 1 << 20, generator=g)
    else:
        t.uniform_(-1.0, 1.0, generator=g)


def _inputs(calls, seed, device="cuda"):
    """Send buffers of every call, and the receive buffers of Bcast, from the seed."""
    g = torch.Generator(device=device).manual_seed(seed)
    sends, recvs = {}, {}
    for key, n in sorted(_layout(calls, 0)[1].items()):
        if n:
            sends[key] = torch.empty(n, dtype=TORCH[key[1]], device=device)
            _fill(sends[key], key[1], g)
    at, total = _layout(calls, 1)
    for key, n in sorted(total.items()):
        if key[0] == "bcast":
            recvs[key] = torch.empty(n, dtype=TORCH[key[1]], device=device)
            _fill(recvs[key], key[1], g)
    for c, (key, start) in zip(calls, at):
        if key in recvs:   # between two calls' buffers: zeros
            end = start + c[1] * _lengths(c)[1]
            recvs[key][end:-(-end // 128) * 128] = 0
    return sends, recvs


def _chain_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    p, n = case["ranks"], case["n"]
    x = torch.empty(p, n, dtype=torch.float64, device="cuda").uniform_(-1.0, 1.0, generator=g)
    return x, n // p   # n is at least p


# ------------------------------------------------------------------ the framework

_mods = {}


def _mod(name):
    if name not in _mods:
        spec = importlib.util.spec_from_file_location(name, os.path.join(ROOT, "dphpc-project_gb300", name + ".py"))
        _mods[name] = sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(_mods[name])
    return _mods[name]


def _api():
    if "lib" not in _mods:
        coll = _mod("gpumpi_coll")
        lib = coll.bind(_mod("gpumpi_host").load_library())
        lib.gpumpi_allreduce_noalloc.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.POINTER(ctypes.c_void_p),
                                                 ctypes.c_int, ctypes.c_uint64, ctypes.c_int, ctypes.c_int,
                                                 ctypes.c_int, ctypes.c_void_p]
        _mods["lib"] = lib
    return _mods["gpumpi_coll"], _mods["lib"]


class State:
    """Buffers, communicators and the plan that a program keeps between calls."""

    def __init__(self, kind):
        self.kind, self.plan, self.comms, self.keep, self.out = kind, None, [], [], None

    def __del__(self):
        if self.plan is not None:
            self.plan.close()
        for c in self.comms:
            c.close()


def _ptrs(t, first, ranks, stride):
    es = t.element_size()
    return [t.data_ptr() + (first + r * stride) * es for r in range(ranks)]


def _descs(coll, s, calls, sends, recvs, comm_of):
    ops = {"bcast": coll.COLL_BCAST, "reduce": coll.COLL_REDUCE, "allreduce": coll.COLL_ALLREDUCE,
           "alltoall": coll.COLL_ALLTOALL, "allgather": coll.COLL_ALLGATHER}
    red = {"sum": coll.OP_SUM, "max": coll.OP_MAX, "min": coll.OP_MIN}
    s_at, r_at = _layout(calls, 0)[0], _layout(calls, 1)[0]
    descs = []
    for c, (ks, fs), (kr, fr) in zip(calls, s_at, r_at):
        kind, p, dt, n, op, root = c
        ns, nr = _lengths(c)
        descs.append(coll.make_desc(comm_of[p], ops[kind], dt, n, _ptrs(sends[ks], fs, p, ns) if ns else None,
                                    _ptrs(recvs[kr], fr, p, nr), red[op], root, s.keep))
    return descs


def prepare(case, seed):
    s = State(case["kind"])
    if case["kind"] == "p2p":
        # the seed gives the number of iterations, whose last one stamps the checked payload
        s.host = _mod("gpumpi_host")
        s.ranks = case["ranks"]
        s.args = ["pairs", "block", str(case["lg_min"]), str(case["lg_max"]), str(case["iters"] + seed % 61)]
        return s
    coll, lib = _api()
    if case["kind"] == "chain":
        return _prepare_chain(s, coll, lib, case, seed)
    calls = _calls(case)
    sends, recvs = _inputs(calls, seed)
    for key, n in _layout(calls, 1)[1].items():
        if key not in recvs:
            recvs[key] = torch.zeros(n, dtype=TORCH[key[1]], device="cuda")
    s.keep += [sends, recvs]
    s.out = {"%s_%s" % k: v for k, v in sorted(recvs.items())}
    if case["kind"] == "noalloc":
        p, n = case["ranks"], case["n"]
        key = ("allreduce", case["dtype"])
        s.lib = lib
        s.args = (coll.ptr_array(_ptrs(sends[key], 0, p, n)), coll.ptr_array(_ptrs(recvs[key], 0, p, n)), p, n,
                  coll.DT[case["dtype"]], coll.OP_SUM, THREADS, None)
        return s
    comm_of = {p: coll.Comm(lib, p) for p in sorted({c[1] for c in calls})}
    s.comms = list(comm_of.values())
    descs = _descs(coll, s, calls, sends, recvs, comm_of)
    s.plan = coll.Plan(lib, descs, threads=THREADS, batched=case["kind"] in ("batch", "host"))
    if case["kind"] == "batch":
        s.plan.capture()
    if case["kind"] == "host":
        _prepare_host(s, calls, sends, recvs)
    return s


def _prepare_host(s, calls, sends, recvs):
    """Pinned host copies of the inputs; the device buffers start out without them."""
    hs = {k: v.cpu().pin_memory() for k, v in sends.items()}
    hb = {k: v.cpu().pin_memory() for k, v in recvs.items() if k[0] == "bcast"}
    hr = {k: torch.zeros(v.numel(), dtype=v.dtype).pin_memory() for k, v in recvs.items()}
    for v in list(sends.values()) + list(recvs.values()):
        v.zero_()
    s.send_ptrs, s.recv_ptrs = [], []
    for c, (ks, fs), (kr, fr) in zip(calls, _layout(calls, 0)[0], _layout(calls, 1)[0]):
        ns, nr = _lengths(c)
        s.send_ptrs += _ptrs(hs[ks], fs, c[1], ns) if ns else _ptrs(hb[kr], fr, c[1], nr)
        s.recv_ptrs += _ptrs(hr[kr], fr, c[1], nr)
    s.keep += [hs, hb]
    s.out = {"%s_%s" % k: v for k, v in sorted(hr.items())}


def _prepare_chain(s, coll, lib, case, seed):
    p, n = case["ranks"], case["n"]
    x, per = _chain_inputs(case, seed)
    total = torch.zeros(p, n, dtype=torch.float64, device="cuda")
    swapped = torch.zeros(p, per * p, dtype=torch.float64, device="cuda")
    joined = torch.zeros(p, per * p, dtype=torch.float64, device="cuda")
    work = torch.zeros(p, n, dtype=torch.float64, device="cuda")
    comm = coll.Comm(lib, p)
    s.comms = [comm]

    def rows(t):
        return _ptrs(t, 0, p, t.shape[1])

    s.plan = coll.Plan(lib, [
        # the sum of every rank's vector, in `work`; every later call reads the one before it
        coll.make_desc(comm, coll.COLL_ALLREDUCE, "float64", n, rows(x), rows(work), coll.OP_SUM, 0, s.keep),
        coll.make_desc(comm, coll.COLL_ALLTOALL, "float64", per, rows(work), rows(swapped), 0, 0, s.keep),
        coll.make_desc(comm, coll.COLL_ALLGATHER, "float64", per, rows(swapped), rows(joined), 0, 0, s.keep),
        coll.make_desc(comm, coll.COLL_REDUCE, "float64", per * p, rows(joined), rows(total), coll.OP_MAX, p - 1,
                       s.keep),
        coll.make_desc(comm, coll.COLL_BCAST, "float64", per * p, None, rows(total), 0, p - 1, s.keep),
    ], threads=THREADS, batched=True)
    s.keep += [x]
    s.out = [work, swapped, joined, total]
    return s


def run(s):
    if s.kind == "p2p":
        r = s.host.run_program("p2p_sweep", s.args, nranks=s.ranks)
        if r.returncode != 0:
            raise RuntimeError(r.stderr[-300:])
        values = []
        for ln in r.lines("p2p "):
            w = ln.split()
            check = int(w[w.index("checksum") + 1], 16)
            values += [int(w[w.index("errors") + 1]), check >> 32, check & 0xffffffff]
        return np.array(values, dtype=np.int64)
    if s.kind == "noalloc":
        rc = s.lib.gpumpi_allreduce_noalloc(*s.args)
        if rc != 0:
            raise RuntimeError("gpumpi_allreduce_noalloc: %d" % rc)
        return s.out
    if s.kind == "host":
        s.plan.run_host(s.send_ptrs, s.recv_ptrs)
        return s.out
    s.plan.launch()
    return s.out


# ------------------------------------------------------------------ bounds

def work(case):
    """Bytes: each input read once, each output written once (host: the same, over the link). Flops: one per folded element."""
    if case["kind"] == "p2p":
        sizes = [1 << lg for lg in range(case["lg_min"], case["lg_max"] + 1)]
        return {"bytes": 2.0 * sum(sizes) * case["iters"] * (case["ranks"] // 2 * 2), "flops": 0.0}
    if case["kind"] == "chain":
        p, n = case["ranks"], case["n"]
        per = n // p
        b = 8 * (2 * p * n + 2 * p * p * per + p * (per + p * per) + (p + 1) * per * p + p * per * p)
        return {"bytes": float(b), "flops": float((p - 1) * (n + per * p))}
    b = f = 0
    for c in _calls(case):
        kind, p, dt, n, _, _ = c
        ns, nr = _lengths(c)
        outs = {"bcast": p - 1, "reduce": 1}.get(kind, p)
        ins = n if kind == "bcast" else p * ns
        b += BYTES[dt] * (ins + outs * nr)
        f += (p - 1) * n if "reduce" in kind else 0
    return {"bytes": float(b), "flops": float(f)}


def exact(case, seed):
    if case["kind"] == "p2p":
        return None
    if case["kind"] == "chain":
        return _exact_chain(case, seed)
    calls = _calls(case)
    sends, recvs = _inputs(calls, seed)
    out = {}
    for key, n in _layout(calls, 1)[1].items():
        if not key[1].startswith("float"):
            out[key] = None
        elif key[0] == "bcast":
            out[key] = recvs[key].double()
        else:
            out[key] = torch.zeros(n, dtype=torch.float64, device="cuda")
    for c, (ks, fs), (kr, fr) in zip(calls, _layout(calls, 0)[0], _layout(calls, 1)[0]):
        kind, p, dt, n, op, root = c
        if out[kr] is None:
            continue
        ns, nr = _lengths(c)
        y = out[kr][fr:fr + p * nr].view(p, nr)
        if kind == "bcast":
            y.copy_(y[root].clone().expand(p, nr))
            continue
        x = sends[ks][fs:fs + p * ns].view(p, ns).double()
        if kind == "alltoall":
            y.view(p, p, n).copy_(x.view(p, p, n).transpose(0, 1))
        elif kind == "allgather":
            y.copy_(x.reshape(1, p * n).expand(p, p * n))
        else:
            r = x.sum(0) if op == "sum" else x.amax(0) if op == "max" else x.amin(0)
            (y if kind == "allreduce" else y[root]).copy_(r)
    return {"%s_%s" % k: v for k, v in sorted(out.items())}


def _exact_chain(case, seed):
    p, n = case["ranks"], case["n"]
    x, per = _chain_inputs(case, seed)
    work = x.sum(0).expand(p, n).contiguous()
    swapped = work[:, :per * p].reshape(p, p, per).transpose(0, 1).reshape(p, per * p).contiguous()
    joined = swapped[:, :per].reshape(1, p * per).expand(p, per * p).contiguous()
    total = torch.zeros(p, n, dtype=torch.float64, device="cuda")
    total[:, :per * p] = joined.amax(0)
    return [work, swapped, joined, total]
