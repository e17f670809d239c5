"""The workloads this engine's speed is judged by, each through its public
Python entry points (osss-ucx_b200/b200shm.py) as a program uses them.

One program: 512 PEs, 160 MiB of symmetric heap each, teams of it at work.
Calls are stream-ordered on the library stream, as in a program that issues
several collectives and then waits once.  Inputs are seeded, with the values
of the repository's configurations: integers uniform in [-1000, 1000] (random
bits for and/or/xor), floats N(0, 1) for SUM, uniform in [-1e6, 1e6) for
MIN/MAX and in [0.999, 1.001) for PROD.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "osss-ucx_b200"))
import b200shm as B  # noqa: E402

NPES = 512
HEAP = 160 << 20
INT_OPS = ["and", "or", "xor", "min", "max", "sum", "prod"]
FLOAT_OPS = ["min", "max", "sum", "prod"]
BATCH_TYPES = ["int32", "int64", "float32", "float64"]
ALGOS = ["linear", "binomial", "rec_dbl", "rabenseifner", "rabenseifner2"]


def listed():
    return [
        # the smallest calls: an int32 sum reduce of 4 KiB per PE, a fcollect
        # of 256 int64 and a barrier, issued in a row by a team of 8
        {"name": "step_8pe", "kind": "step", "pes": 8, "nelems": 1024, "blocks": 256},
        # an everyday all-reduce: 32 KiB vectors over a node-sized team
        {"name": "reduce_f32_32x8192", "kind": "reduce", "pes": 32, "nelems": 8192,
         "dtype": "float32", "op": "sum", "algo": "rec_dbl", "src_shift": 0, "dst_shift": 0},
        # the largest: the three headline reductions, 64 PEs x 2^20 elements
        {"name": "headline_64x1Mi", "kind": "headline", "pes": 64, "nelems": 1 << 20,
         "algo": "rec_dbl"},
        # a ragged one: 100 PEs, an odd count, part of a vector that begins
        # off the 16-byte grid (an array slice passed as source and dest)
        {"name": "reduce_f64_100x50001", "kind": "reduce", "pes": 100, "nelems": 50001,
         "dtype": "float64", "op": "sum", "algo": "rabenseifner", "src_shift": 1, "dst_shift": 1},
        # data movement at the sizes of the 128-PE configuration
        {"name": "fcollect_128x32KiB", "kind": "fcollect", "pes": 128, "nbytes": 32768},
        {"name": "alltoall_128x64KiB", "kind": "alltoall", "pes": 128, "nbytes": 65536},
        {"name": "alltoalls_128x4096", "kind": "alltoalls", "pes": 128, "nelems": 4096,
         "esize": 8, "dst": 2, "sst": 3},
        # an all-to-all of records whose size is no power of two (251 int32)
        {"name": "alltoall_96x1004B", "kind": "alltoall", "pes": 96, "nbytes": 1004},
        # uneven contributions: on average 8192 int32 of each of 64 PEs
        {"name": "collect_64_uneven", "kind": "collect", "pes": 64, "mean": 8192, "esize": 4},
        # 2^20 atomic fetch-adds on random PEs and offsets
        {"name": "amo_fetch_add_1Mi", "kind": "amo", "pes": 128, "counters": 1 << 20,
         "nops": 1 << 20, "amo": "fetch_add", "dtype": "int64"},
        # batching: 2048 reductions of uneven size over 256 teams, one graph
        {"name": "batch_2048", "kind": "batch", "teams": 256, "reductions": 2048,
         "most": 1 << 16},
        # serving: a burst of 2048 mixed requests through the serving loop
        {"name": "serve_2048", "kind": "serve", "requests": 2048, "most": 1 << 18},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "reduce", "reduce", "headline", "fcollect", "alltoall",
                       "alltoalls", "collect", "amo", "batch", "serve"])
    if kind == "step":
        return {"kind": kind, "pes": log(2, 64), "nelems": log(1, 4096), "blocks": log(1, 512)}
    if kind == "reduce":
        dt = rng.choice(["uint8", "int16", "int32", "int64", "float32", "float64", "complex64",
                         "complex128"])
        op = rng.choice(INT_OPS if "int" in dt else ["sum", "prod"] if dt[0] == "c" else FLOAT_OPS)
        pes = log(2, 256)
        es = np.dtype(dt).itemsize
        n = log(16, min(1 << 20, (256 << 20) // (pes * es)))
        shift = rng.choice([0, 0, 0, 1, 3])
        return {"kind": kind, "pes": pes, "nelems": n, "dtype": dt, "op": op,
                "algo": rng.choice(ALGOS), "src_shift": shift,
                "dst_shift": rng.choice([shift, shift, 0])}
    if kind == "headline":
        return {"kind": kind, "pes": rng.choice([16, 24, 32, 48, 64]), "nelems": log(1 << 16, 1 << 20),
                "algo": rng.choice(["rec_dbl", "rabenseifner"])}
    if kind == "fcollect":
        pes = log(4, 128)
        return {"kind": kind, "pes": pes, "nbytes": log(1, 64) * rng.choice([4, 8, 16, 512])}
    if kind == "alltoall":
        pes = log(4, 128)
        return {"kind": kind, "pes": pes, "nbytes": log(1, 4096) * rng.choice([4, 8, 16])}
    if kind == "alltoalls":
        return {"kind": kind, "pes": log(4, 128), "nelems": log(1, 4096), "esize": rng.choice([4, 8]),
                "dst": rng.choice([1, 2, 3]), "sst": rng.choice([1, 2, 3])}
    if kind == "collect":
        return {"kind": kind, "pes": log(4, 128), "mean": log(1, 8192), "esize": rng.choice([4, 8])}
    if kind == "amo":
        return {"kind": kind, "pes": log(8, 128), "counters": log(1 << 16, 1 << 20),
                "nops": log(1 << 8, 1 << 19), "amo": rng.choice(["fetch_add", "add", "swap", "xor"]),
                "dtype": rng.choice(["int32", "int64"])}
    if kind == "batch":
        return {"kind": kind, "teams": log(32, 256), "reductions": log(64, 2048),
                "most": log(1 << 12, 1 << 16)}
    return {"kind": kind, "requests": log(256, 2048), "most": log(1 << 12, 1 << 18)}


# ---- what a program keeps ---------------------------------------------------

class Objects:
    """Symmetric objects of one workload, freed when nothing refers to them."""

    def __init__(self):
        if not B.initialized():
            B.init(NPES, HEAP)
        self.offs = []

    def malloc(self, nbytes):
        self.offs.append(B.malloc(max(int(nbytes), 1)))
        return self.offs[-1]

    def __del__(self):
        for off in self.offs:
            B.free(off)


class Rows:
    """An element range of a symmetric object in every member of a team, as a
    [members, elements] array of the device; it keeps the object alive."""

    def __init__(self, objects, off, team, n, dtype):
        start, stride, size = team
        dt = np.dtype(dtype)
        self.objects = objects
        self.__cuda_array_interface__ = {
            "shape": (size, n), "typestr": dt.str, "version": 3, "data": (B.ptr(start, off), False),
            "strides": (stride * B.heap_slice(), dt.itemsize)}


class State:
    """What one workload keeps: its symmetric objects, views of them, a plan."""

    def __init__(self, case):
        self.case, self.objects = case, Objects()
        self.malloc = self.objects.malloc

    def rows(self, off, team, n, dtype):
        return torch.as_tensor(Rows(self.objects, off, team, n, dtype), device="cuda")


_server = []


def server():
    """The program's one serving loop."""
    if not _server:
        _server.append(B.Server(queue_slots=256, idle_seconds=0.001))
    return _server[0]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _values(shape, dtype, op, g):
    dt = getattr(torch, dtype)
    if op in ("and", "or", "xor", "bits"):
        b = torch.randint(0, 256, tuple(shape[:-1]) + (shape[-1] * dt.itemsize,), dtype=torch.uint8,
                          device="cuda", generator=g)
        return b.view(dt)
    if not (dt.is_floating_point or dt.is_complex):
        lo, hi = (0, 256) if dtype == "uint8" else (-1000, 1001)
        return torch.randint(lo, hi, shape, dtype=torch.int32, device="cuda", generator=g).to(dt)
    if op == "sum":
        return torch.randn(shape, dtype=dt, device="cuda", generator=g)
    if dt.is_complex:
        real = torch.float32 if dt == torch.complex64 else torch.float64
        u = torch.rand(tuple(shape) + (2,), dtype=real, device="cuda", generator=g) - 0.5
        return torch.view_as_complex(u * 0.002) + 1
    u = torch.rand(shape, dtype=dt, device="cuda", generator=g)
    return u * 0.002 + 0.999 if op == "prod" else u * 2e6 - 1e6


def _reduced(x, op):
    """The reduction over rows, in 64 bits (integers wrap at their own width)."""
    if op in ("and", "or", "xor"):
        r = x[0].clone()
        for row in x[1:]:
            r = r & row if op == "and" else r | row if op == "or" else r ^ row
        return r
    if x.dtype.is_complex:
        wide = x.to(torch.complex128)
    else:
        wide = x.to(torch.float64 if x.dtype.is_floating_point else torch.int64)
    r = {"sum": lambda: wide.sum(0), "prod": lambda: wide.prod(0),
         "min": lambda: wide.amin(0), "max": lambda: wide.amax(0)}[op]()
    return r if x.dtype.is_floating_point or x.dtype.is_complex else r.to(x.dtype)


# ---- the workloads ------------------------------------------------------------
# Each kind: its inputs as plain tensors, made from the seed alone; their
# placing in the symmetric heap; the pass; the bytes and operations of a pass;
# the expected outputs.

def _team(case):
    return (0, 1, case["pes"])


HEADLINE = [("sum", "float32"), ("max", "float64"), ("xor", "int64")]


def _step_inputs(c, seed):
    g = _generator(seed)
    return [_values((c["pes"], c["nelems"]), "int32", "sum", g),
            _values((c["pes"], c["blocks"]), "int64", "sum", g)]


def _prepare_step(s, c, seed):
    x, y = _step_inputs(c, seed)
    t, P = _team(c), c["pes"]
    s.src, s.dst = s.malloc(4 * c["nelems"]), s.malloc(4 * c["nelems"])
    s.fsrc, s.fdst = s.malloc(8 * c["blocks"]), s.malloc(8 * c["blocks"] * P)
    s.rows(s.src, t, c["nelems"], "int32").copy_(x)
    s.rows(s.fsrc, t, c["blocks"], "int64").copy_(y)
    s.out = [s.rows(s.dst, t, c["nelems"], "int32"), s.rows(s.fdst, t, c["blocks"] * P, "int64")]


def _run_step(s, c):
    t, stream = _team(c), B.stream()
    B.reduce("sum", "int32", "rec_dbl", s.dst, s.src, c["nelems"], team=t, stream=stream)
    B.fcollect(s.fdst, s.fsrc, 8 * c["blocks"], team=t, stream=stream)
    B.barrier("binomial_tree", team=t, stream=stream)


def _exact_step(c, seed):
    x, y = _step_inputs(c, seed)
    return [_reduced(x, "sum").expand(c["pes"], -1), y.reshape(1, -1).expand(c["pes"], -1)]


def _work_step(c):
    P = c["pes"]
    return {"bytes": P * (8 * c["nelems"] + 8 * c["blocks"] * (1 + P)), "flops": (P - 1) * c["nelems"]}


def _reductions(c):
    """(op, dtype, algo, src_shift, dst_shift) of the reductions of a pass."""
    if c["kind"] == "headline":
        return [(op, dt, c["algo"], 0, 0) for op, dt in HEADLINE]
    return [(c["op"], c["dtype"], c["algo"], c["src_shift"], c["dst_shift"])]


def _reduce_inputs(c, seed):
    g = _generator(seed)
    return [_values((c["pes"], c["nelems"]), dt, op, g) for op, dt, *_ in _reductions(c)]


def _prepare_reduce(s, c, seed):
    s.calls, s.out = [], []
    for (op, dt, algo, a, b), x in zip(_reductions(c), _reduce_inputs(c, seed)):
        es, n = np.dtype(dt).itemsize, c["nelems"]
        src = s.malloc((n + a) * es) + a * es
        dst = s.malloc((n + b) * es) + b * es
        s.rows(src, _team(c), n, dt).copy_(x)
        s.calls.append((op, dt, algo, dst, src))
        s.out.append(s.rows(dst, _team(c), n, dt))


def _run_reduce(s, c):
    for op, dt, algo, dst, src in s.calls:
        B.reduce(op, dt, algo, dst, src, c["nelems"], team=_team(c), stream=B.stream())


def _exact_reduce(c, seed):
    return [_reduced(x, op).expand(c["pes"], -1)
            for (op, *_), x in zip(_reductions(c), _reduce_inputs(c, seed))]


def _work_reduce(c):
    P, n = c["pes"], c["nelems"]
    return {"bytes": sum(2 * P * n * np.dtype(dt).itemsize for _, dt, *_ in _reductions(c)),
            "flops": len(_reductions(c)) * (P - 1) * n}


def _counts(c):
    return np.random.default_rng(c["pes"] * 1000003 + c["mean"]).integers(0, 2 * c["mean"] + 1, c["pes"])


def _copy_inputs(c, seed):
    """Rows of bytes (fcollect, alltoall), of elements (alltoalls), or rows of
    elements and how many of them each member contributes (collect; fixed for
    a case)."""
    g, P = _generator(seed), c["pes"]
    if c["kind"] == "fcollect":
        return _values((P, c["nbytes"]), "uint8", "bits", g)
    if c["kind"] == "alltoall":
        return _values((P, P * c["nbytes"]), "uint8", "bits", g)
    if c["kind"] == "alltoalls":
        return _values((P, (P * c["nelems"] - 1) * c["sst"] + 1), "int%d" % (8 * c["esize"]), "bits", g)
    return _values((P, 2 * c["mean"]), "int%d" % (8 * c["esize"]), "bits", g), _counts(c)


def _prepare_copy(s, c, seed):
    t, P, kind = _team(c), c["pes"], c["kind"]
    x = _copy_inputs(c, seed)
    if kind == "collect":
        x, counts = x
        s.sizes = (counts * c["esize"]).astype(np.uint64)
        n = max(int(counts.sum()), 1)
    else:
        n = {"fcollect": lambda: P * c["nbytes"], "alltoall": lambda: P * c["nbytes"],
             "alltoalls": lambda: (P * c["nelems"] - 1) * c["dst"] + 1}[kind]()
    dt = str(x.dtype).split(".")[1]
    s.src, s.dst = s.malloc(x.shape[1] * x.itemsize), s.malloc(n * x.itemsize)
    s.rows(s.src, t, x.shape[1], dt).copy_(x)
    s.out = [s.rows(s.dst, t, n, dt).zero_()]


def _run_copy(s, c):
    t, stream, kind = _team(c), B.stream(), c["kind"]
    if kind == "fcollect":
        B.fcollect(s.dst, s.src, c["nbytes"], team=t, stream=stream)
    elif kind == "alltoall":
        B.alltoall(s.dst, s.src, c["nbytes"], team=t, stream=stream)
    elif kind == "alltoalls":
        B.alltoalls(s.dst, s.src, c["dst"], c["sst"], c["nelems"], c["esize"], team=t, stream=stream)
    else:
        B.collect(s.dst, s.src, s.sizes, team=t, stream=stream)


def _exact_copy(c, seed):
    P, kind = c["pes"], c["kind"]
    x = _copy_inputs(c, seed)
    if kind == "fcollect":
        return [x.reshape(1, -1).expand(P, -1)]
    if kind == "alltoall":
        return [x.reshape(P, P, -1).transpose(0, 1).reshape(P, -1)]
    if kind == "alltoalls":
        y = x[:, ::c["sst"]].reshape(P, P, -1).transpose(0, 1).reshape(P, -1)
        out = torch.zeros((P, (P * c["nelems"] - 1) * c["dst"] + 1), dtype=x.dtype, device="cuda")
        out[:, ::c["dst"]] = y
        return [out]
    x, counts = x
    y = torch.cat([row[:int(k)] for row, k in zip(x, counts)])
    return [(y if len(y) else x.new_zeros(1)).expand(P, -1)]


def _work_copy(c):
    P, kind = c["pes"], c["kind"]
    if kind == "alltoall":
        n = 2 * P * P * c["nbytes"]
    elif kind == "alltoalls":
        n = 2 * P * P * c["nelems"] * c["esize"]
    else:
        mine = P * c["nbytes"] if kind == "fcollect" else int(_counts(c).sum()) * c["esize"]
        n = (1 + P) * mine
    return {"bytes": n, "flops": 0}


def _amo_inputs(c, seed):
    """Counters, and operations on random ones.  Every operation has a counter
    of its own, so the old values do not depend on the order of execution."""
    g, P, n = _generator(seed), c["pes"], min(c["nops"], c["pes"] * c["counters"])
    x = _values((P, c["counters"]), c["dtype"], "sum", g)
    at = torch.randperm(P * c["counters"], device="cuda", generator=g)[:n]
    return x, at, _values((n,), c["dtype"], "sum", g)


def _prepare_amo(s, c, seed):
    x, at, s.value = _amo_inputs(c, seed)
    es = np.dtype(c["dtype"]).itemsize
    s.obj = s.malloc(c["counters"] * es)
    counters = s.rows(s.obj, _team(c), c["counters"], c["dtype"])
    counters.copy_(x)
    s.pe = (at // c["counters"]).to(torch.int32)
    s.off = at % c["counters"] * es + s.obj
    s.fetched = torch.zeros_like(s.value)
    s.out = [counters, s.fetched]


def _run_amo(s, c):
    old = s.fetched.data_ptr() if c["amo"] in ("fetch_add", "swap") else None
    B.amo_batch(c["amo"], c["dtype"], s.value.numel(), s.pe.data_ptr(), s.off.data_ptr(),
                s.value.data_ptr(), None, old, stream=B.stream())


def _exact_amo(c, seed):
    x, at, v = _amo_inputs(c, seed)
    flat = x.reshape(-1)
    old = flat[at]
    flat[at] = {"fetch_add": old + v, "add": old + v, "swap": v, "xor": old ^ v}[c["amo"]]
    return [x, old if c["amo"] in ("fetch_add", "swap") else torch.zeros_like(v)]


def _work_amo(c):
    n, es = min(c["nops"], c["pes"] * c["counters"]), np.dtype(c["dtype"]).itemsize
    fetch = c["amo"] in ("fetch_add", "swap")
    return {"bytes": n * (12 + es * (4 if fetch else 3)), "flops": n}


def _place(top, pes, nbytes):
    """An offset free in all of `pes` (top: first free byte of each PE)."""
    off = int(top[pes].max())
    top[pes] = off + (nbytes + 255) // 256 * 256
    return off


def _batch_plan(c):
    """Teams of uneven size (power law in [2, 256], strides 1, 2, 4) and
    reductions over them, nelems log-uniform in [16, most]; every type has
    its own source and dest object.  Fixed for a case: a program's plan."""
    rng = np.random.default_rng(c["teams"] * 1000003 + c["reductions"])
    teams, pos = [], 0
    for k in range(c["teams"]):
        size = int(np.clip(1 / (0.5 - rng.random() * (0.5 - 1 / 256)), 2, 256))
        stride = [1, 2, 4][k % 3]
        while (size - 1) * stride + 1 > NPES:
            stride //= 2
        span = (size - 1) * stride + 1
        teams.append((pos % (NPES - span + 1), stride, size))
        pos += span
    top = {dt: np.zeros(NPES, np.int64) for dt in BATCH_TYPES}
    items = []
    for _ in range(c["reductions"]):
        team = teams[int(rng.integers(len(teams)))]
        n = int(math.exp(rng.uniform(math.log(16), math.log(c["most"]))))
        dt = BATCH_TYPES[int(rng.integers(4))]
        ops = INT_OPS if "int" in dt else FLOAT_OPS
        pes = team[0] + np.arange(team[2]) * team[1]
        off = _place(top[dt], pes, n * np.dtype(dt).itemsize)
        items.append(dict(op=ops[int(rng.integers(len(ops)))], dtype=dt, algo="rec_dbl", team=team,
                          nelems=n, off=off))
    return items, {dt: max(int(v.max()), 256) for dt, v in top.items()}


def _item_rows(view, item):
    """The item's part of a [PEs, elements] array of its type."""
    start, stride, size = item["team"]
    first = item["off"] // np.dtype(item["dtype"]).itemsize
    return view[start:start + (size - 1) * stride + 1:stride, first:first + item["nelems"]]


def _prepare_batch(s, c, seed):
    items, size = _batch_plan(c)
    g, whole = _generator(seed), (0, 1, NPES)
    src, dst, views = {}, {}, {}
    for dt, nbytes in size.items():
        n = nbytes // np.dtype(dt).itemsize
        src[dt], dst[dt] = s.malloc(nbytes), s.malloc(nbytes)
        views[dt] = s.rows(src[dt], whole, n, dt)
    s.out = [s.rows(dst[dt], whole, size[dt] // np.dtype(dt).itemsize, dt).zero_() for dt in size]
    for it in items:
        v = _item_rows(views[it["dtype"]], it)
        v.copy_(_values(tuple(v.shape), it["dtype"], it["op"], g))
    descs = B.make_descs([dict(it, src=src[it["dtype"]] + it["off"], dest=dst[it["dtype"]] + it["off"])
                          for it in items])
    s.batch = B.Batch(descs, B.BATCH_NO_TUNE | B.BATCH_GRAPH)


def _run_batch(s, c):
    s.batch.run(stream=B.stream())


def _exact_batch(c, seed):
    items, size = _batch_plan(c)
    g = _generator(seed)
    out = {dt: torch.zeros((NPES, n // np.dtype(dt).itemsize), dtype=getattr(torch, dt), device="cuda")
           for dt, n in size.items()}
    out["float32"] = out["float32"].double()
    for it in items:
        v = _item_rows(out[it["dtype"]], it)
        v.copy_(_reduced(_values(tuple(v.shape), it["dtype"], it["op"], g), it["op"]).expand(v.shape))
    return [out[dt] for dt in size]


def _work_batch(c):
    items, _ = _batch_plan(c)
    return {"bytes": sum(2 * i["team"][2] * i["nelems"] * np.dtype(i["dtype"]).itemsize for i in items),
            "flops": sum((i["team"][2] - 1) * i["nelems"] for i in items)}


SERVE_PES = 256
SERVE_SRC = 1 << 20  # bytes of every PE's source object, 8-byte words
KINDS = ["reduce", "fcollect", "alltoall", "put", "get", "amo"]


def _serve_plan(c):
    """Requests of 64 teams of 4 PEs: kinds uniform, payload (bytes received
    per PE) log-uniform in [8, most].  Reductions have a dest object per
    type, copies one of bytes, atomics (fetch-adds) a counter each."""
    rng = np.random.default_rng(c["requests"] * 1000003 + c["most"])
    top = {dt: np.zeros(SERVE_PES, np.int64) for dt in BATCH_TYPES + ["uint8"]}
    items = []
    for k in range(c["requests"]):
        kind = KINDS[int(rng.integers(6))]
        team = (4 * int(rng.integers(SERVE_PES // 4)), 1, 4)
        nb = int(math.exp(rng.uniform(math.log(8), math.log(c["most"]))))
        dt = BATCH_TYPES[int(rng.integers(4))] if kind == "reduce" else "uint8"
        es = np.dtype(dt).itemsize
        it = dict(kind=kind, team=team, dtype=dt, op="sum", at=int(rng.integers(SERVE_SRC // 2 // 16)) * 16)
        if kind == "amo":
            it.update(pe=team[0], off=8 * k, value=int(rng.integers(1, 1000)), nelems=0)
        else:
            n = max(nb // es if kind == "reduce" else nb // (1 if kind in ("put", "get") else 4), 1)
            span = n * es * (4 if kind in ("fcollect", "alltoall") else 1)
            pes = np.arange(team[0], team[0] + 4)
            it.update(nelems=n, off=_place(top[dt], pes, span), span=span,
                      pe=team[0] + int(rng.integers(1, 4)))
        items.append(it)
    return items, {dt: max(int(v.max()), 256) for dt, v in top.items()}


def _serve_inputs(c, seed):
    g = _generator(seed)
    x = {dt: _values((SERVE_PES, SERVE_SRC // np.dtype(dt).itemsize), dt, "sum", g) for dt in BATCH_TYPES}
    x["uint8"] = _values((SERVE_PES, SERVE_SRC), "uint8", "bits", g)
    return x, _values((SERVE_PES, c["requests"]), "int64", "sum", g)


def _prepare_serve(s, c, seed):
    items, size = _serve_plan(c)
    x, counters = _serve_inputs(c, seed)
    team = (0, 1, SERVE_PES)
    src = {dt: s.malloc(SERVE_SRC) for dt in size}
    dst = {dt: s.malloc(n) for dt, n in size.items()}
    ctr = s.malloc(8 * c["requests"])
    for dt in size:
        s.rows(src[dt], team, x[dt].shape[1], dt).copy_(x[dt])
    out = [s.rows(dst[dt], team, size[dt] // np.dtype(dt).itemsize, dt).zero_() for dt in size]
    words = s.rows(ctr, team, c["requests"], "int64")
    words.copy_(counters)
    reqs = []
    for it in items:
        if it["kind"] == "amo":
            reqs.append(dict(kind="amo", op="fetch_add", dtype="int64", pe=it["pe"], dest=ctr + it["off"],
                             value=it["value"]))
        else:
            team4 = it["team"] if it["kind"] not in ("put", "get") else (it["team"][0], 1, 1)
            reqs.append(dict(kind=it["kind"], op="sum", dtype=it["dtype"], team=team4, pe=it["pe"],
                             dest=dst[it["dtype"]] + it["off"], src=src[it["dtype"]] + it["at"],
                             n=it["nelems"]))
    s.reqs, s.arrival = B.make_requests(reqs), np.zeros(len(reqs))
    s.amos = np.array([it["kind"] == "amo" for it in items])
    s.out = out + [words]


def _run_serve(s, c):
    _, fetched = B.replay(s.reqs, s.arrival, server())
    return s.out + [fetched[s.amos].view(np.int64)]


def _exact_serve(c, seed):
    items, size = _serve_plan(c)
    x, words = _serve_inputs(c, seed)
    out = {dt: torch.zeros((SERVE_PES, n // np.dtype(dt).itemsize), dtype=getattr(torch, dt), device="cuda")
           for dt, n in size.items()}
    out["float32"] = out["float32"].double()
    olds = []
    for it in items:
        t0, n, es = it["team"][0], it["nelems"], np.dtype(it["dtype"]).itemsize
        a, o = it["at"] // es, it["off"] // es
        src, dst = x[it["dtype"]][t0:t0 + 4], out[it["dtype"]][t0:t0 + 4]
        if it["kind"] == "reduce":
            dst[:, o:o + n] = _reduced(src[:, a:a + n], "sum")
        elif it["kind"] == "fcollect":
            dst[:, o:o + 4 * n] = src[:, a:a + n].reshape(-1)
        elif it["kind"] == "alltoall":
            dst[:, o:o + 4 * n] = src[:, a:a + 4 * n].reshape(4, 4, n).transpose(0, 1).reshape(4, -1)
        elif it["kind"] == "put":
            dst[it["pe"] - t0, o:o + n] = src[0, a:a + n]
        elif it["kind"] == "get":
            dst[0, o:o + n] = src[it["pe"] - t0, a:a + n]
        else:
            w = words[it["pe"], it["off"] // 8]
            olds.append(w.clone())
            w += it["value"]
    olds = torch.stack(olds) if olds else torch.zeros(0, dtype=torch.int64)
    return [out[dt] for dt in size] + [words, olds]


def _work_serve(c):
    n = flops = 0
    for it in _serve_plan(c)[0]:
        k = it["nelems"] * np.dtype(it["dtype"]).itemsize
        n += {"reduce": 8 * k, "fcollect": 20 * k, "alltoall": 32 * k, "put": 2 * k, "get": 2 * k,
              "amo": 16}[it["kind"]]
        flops += 3 * it["nelems"] if it["kind"] == "reduce" else 0
    return {"bytes": n, "flops": flops}


_FAMILY = {"step": (_prepare_step, _run_step, _work_step, _exact_step),
           "reduce": (_prepare_reduce, _run_reduce, _work_reduce, _exact_reduce),
           "headline": (_prepare_reduce, _run_reduce, _work_reduce, _exact_reduce),
           "fcollect": (_prepare_copy, _run_copy, _work_copy, _exact_copy),
           "alltoall": (_prepare_copy, _run_copy, _work_copy, _exact_copy),
           "alltoalls": (_prepare_copy, _run_copy, _work_copy, _exact_copy),
           "collect": (_prepare_copy, _run_copy, _work_copy, _exact_copy),
           "amo": (_prepare_amo, _run_amo, _work_amo, _exact_amo),
           "batch": (_prepare_batch, _run_batch, _work_batch, _exact_batch),
           "serve": (_prepare_serve, _run_serve, _work_serve, _exact_serve)}


def prepare(case, seed):
    s = State(case)
    _FAMILY[case["kind"]][0](s, case, seed)
    torch.cuda.synchronize()
    return s


def run(state):
    got = _FAMILY[state.case["kind"]][1](state, state.case)
    return state.out if got is None else got


def work(case):
    return _FAMILY[case["kind"]][2](case)


def exact(case, seed):
    return _FAMILY[case["kind"]][3](case, seed)
