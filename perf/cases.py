"""The work a program does with this library, at the sizes it does it.

`listed()` names the cases, `draw(rng)` gives one more of the same ranges, `prepare` builds what
the program holds before the call (a context with the graph's store on the device, plans as C
arrays, tables, pinned buffers), `run` makes one pass through the public entry points and
`work` says what that pass cannot do without.

Graphs are the generator's (organisations, units, persons, courses, documents), from 20
organisations (2.8e5 triples) to 10,000 (1.37e8 triples), uniform or with Zipf-drawn hubs.  A
case's graph, constants and row choices are its own; the seed says where its vertex ids begin (as
a dataset loaded behind others), what a table's bystander columns hold and in what order requests
arrive, so a case's results have one shape and every seed's are others.  All results are ids,
compared whole; none is a computed number, so `exact` has no values to give.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "wukong-cube_b200"))
import workloads  # noqa: E402
import wukong_b200 as wk  # noqa: E402

# means of the generator, per organisation
UNITS, PERSONS, PERSONS_A, TRIPLES = 20, 900, 300, 13650
TAKES = 5.0          # courses per person
STORE_BYTES = 152    # store bytes per triple at the default load factor


def listed():
    return [
        # one selective query, answer wanted on the host: the smallest call, all latency
        {"name": "chain_host_20", "kind": "query", "query": "chain", "orgs": 20, "zipf": False, "mode": "resident"},
        # non-selective queries from the type index, table kept on the device for what follows
        {"name": "star_1000", "kind": "query", "query": "star", "orgs": 1000, "zipf": False, "mode": "resident"},
        # the same plan asked again and again (captured graph), on a graph with hub vertices
        {"name": "star_zipf_3001", "kind": "query", "query": "star", "orgs": 3001, "zipf": True, "mode": "graph"},
        # three joins from a predicate index, two of them on functional predicates; the largest graph
        {"name": "triangle_10000", "kind": "query", "query": "triangle", "orgs": 10000, "zipf": False, "mode": "resident"},
        # a handful of light queries collected by a front end, answers on the host
        {"name": "batch_64", "kind": "batch", "n": 64, "stream": 0, "orgs": 200, "zipf": False},
        # a full batch of light queries of 2 to 6 patterns, answers on the host
        {"name": "batch_16384", "kind": "batch", "n": 16384, "stream": 0, "orgs": 2000, "zipf": False},
        # consecutive full batches, pipelined, on a graph with hub vertices
        {"name": "stream_49152_zipf", "kind": "batch", "n": 49152, "stream": 16384, "orgs": 1501, "zipf": True},
        # one expansion of a program's own table, rows in no order, an odd row count
        {"name": "expand_1000003", "kind": "step", "op": "k2u", "rows": 1000003, "cols": 2, "orgs": 1000, "zipf": False},
        # one membership filter of a program's own table, rows in no order
        {"name": "filter_2500001", "kind": "step", "op": "k2k", "rows": 2500001, "cols": 3, "orgs": 700, "zipf": False},
        # DISTINCT and the projection over a large table in no order
        {"name": "distinct_3000000", "kind": "final", "rows": 3000000, "cols": 3, "keep": 2, "orgs": 700, "zipf": False},
        # a dataset loaded and its first query answered
        {"name": "build_500", "kind": "build", "orgs": 500, "zipf": False, "versatile": False},
        # a burst of requests, 2% of them heavy, through the serving loop, row counts back
        {"name": "serve_4096", "kind": "serve", "n": 4096, "orgs": 200, "zipf": False, "heavy": 0.02},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "query", "batch", "batch", "step", "step", "final", "build", "serve"])
    zipf = rng.random() < 0.3
    if kind == "query":
        q = rng.choice(["chain", "star", "triangle", "light"])
        return {"kind": kind, "query": q, "orgs": _log(rng, 20, 2500), "zipf": zipf,
                "mode": rng.choice(["plain", "resident", "graph"])}
    if kind == "batch":
        n = _log(rng, 16, 20000)
        return {"kind": kind, "n": n, "stream": rng.choice([0, 0, max(8, n // rng.randint(2, 5))]),
                "orgs": _log(rng, 20, 1500), "zipf": zipf}
    if kind == "step":
        return {"kind": kind, "op": rng.choice(["k2u", "k2k", "k2c", "kuu"]), "rows": _log(rng, 1000, 2500000),
                "cols": rng.randint(2, 5), "orgs": _log(rng, 20, 1000), "zipf": zipf}
    if kind == "final":
        cols = rng.randint(2, 5)
        return {"kind": kind, "rows": _log(rng, 1000, 3000000), "cols": cols, "keep": rng.randint(1, cols),
                "orgs": _log(rng, 20, 700), "zipf": zipf}
    if kind == "build":
        return {"kind": kind, "orgs": _log(rng, 20, 700), "zipf": zipf, "versatile": rng.random() < 0.4}
    return {"kind": "serve", "n": _log(rng, 256, 4000), "orgs": _log(rng, 20, 190), "zipf": zipf,
            "heavy": rng.choice([0.0, 0.01, 0.02])}


class _Device:
    """A device array by its address, for torch.as_tensor; it keeps what owns the memory."""

    def __init__(self, owner, ptr, rows, cols):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (rows, cols), "typestr": "<i4", "data": (ptr, False), "version": 3}


class State:
    """What a program holds: a context, its store, plans and buffers.  Closed when dropped."""

    def __init__(self, case, seed):
        self.kind = case["kind"]
        self.lib = wk.lib()
        self.ctx = wk.Context(0)
        self.tables = []
        self.triples, self.v = wk.synth_generate(case["orgs"], seed=0, zipf=case["zipf"])
        shift = 1 + seed * 7919 % (1 << 20)
        first = self.v["first_vid"]
        self.triples[:, 0] += np.uint32(shift)
        o = self.triples[:, 2]
        o += (o >= first).astype(np.uint32) * np.uint32(shift)
        self.v = dict(self.v, first_vid=first + shift, next_vid=self.v["next_vid"] + shift)

    def build(self, versatile=False):
        self.ctx.build_store(self.triples, versatile=versatile)
        self.triples = None

    def index(self, tid):
        """The vertices of a type, from the store's index."""
        t = self.ctx.table()
        self.ctx.index_to_unknown(tid, wk.IN, t)
        got = t.download().reshape(-1)
        t.free()
        return got

    def plan(self, q):
        self.q = q.as_c()
        self.mode = wk.MODE_RESIDENT
        self.v2c = (C.c_int32 * max(q.nvars, 1))()
        self.cols, self.rows, self.table = C.c_int32(), C.c_uint64(), C.c_void_p()

    def check(self, rc):
        if rc:
            wk._check(rc, self.ctx.h)

    def device_table(self, table):
        """A result table where it is, on the device."""
        rows, cols, ptr = C.c_uint64(), C.c_int32(), C.c_void_p()
        self.check(self.lib.wk_table_shape(self.ctx.h, table, C.byref(rows), C.byref(cols)))
        if not rows.value:
            return torch.empty((0, cols.value), dtype=torch.int32, device="cuda")
        self.check(self.lib.wk_table_device_ptr(self.ctx.h, table, C.byref(ptr)))
        return torch.as_tensor(_Device(self, ptr.value, rows.value, cols.value), device="cuda")

    def pinned(self, elems):
        self.out_t = torch.empty(elems, dtype=torch.int32, pin_memory=True)
        self.out = self.out_t.numpy()
        self.out_ptr = C.c_void_p(self.out_t.data_ptr())

    def __del__(self):
        if getattr(self, "ctx", None) is not None:
            for t in self.tables:
                t.free()
            self.ctx.close()


def _light(s, n, min_len=2):
    inst = {t: s.index(t) for t in range(s.v["t_org"], s.v["t_doc"] + 1)}
    return workloads.light_queries(s.v, inst, n, seed=1, min_len=min_len)


RESULT = np.dtype([("rows", "<u8"), ("elem_offset", "<u8"), ("cols", "<i4"), ("status", "<i4"),
                   ("t_arrive_us", "<f8"), ("t_done_us", "<f8")])


def _prepare_query(s, case, rng, seed):
    s.build()
    v = s.v
    if case["query"] == "chain":
        units = s.index(v["t_unit"])
        q = workloads.small_chain(v, int(units[rng.integers(len(units))]))
    elif case["query"] == "light":
        q = _light(s, 1, min_len=6)[0]
    else:
        q = workloads.heavy_star(v) if case["query"] == "star" else workloads.heavy_triangle(v)
    s.plan(q)
    s.host = case["query"] in ("chain", "light")
    s.mode = {"plain": wk.MODE_PLAIN, "resident": wk.MODE_RESIDENT, "graph": wk.MODE_GRAPH}[case["mode"]]
    if s.host:
        # the largest table that one constant of these graphs reaches is the Zipf hub's
        s.pinned(1 << 22)


def _prepare_batch(s, case, rng, seed):
    s.build()
    qs = _light(s, case["n"])
    s.qs, s.keep = wk.queries_as_c(qs)
    s.n, s.stream = case["n"], case["stream"]
    s.res = (wk.QResult * s.n)()
    # room for the tables: 4 KB a query on average and a few hub tables
    s.pinned(s.n * 1024 + (1 << 23))


def _prepare_step(s, case, rng, seed):
    s.op = case["op"]
    s.build(versatile=s.op == "kuu")
    v, R, cols = s.v, case["rows"], case["cols"]
    persons = np.concatenate([s.index(v[k]) for k in ("t_person_a", "t_person_b", "t_person_c")])
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    p = torch.from_numpy(persons.astype(np.int64)).cuda()
    rows = torch.randint(0, 1 << 30, (R, cols), generator=g, device="cuda")
    g.manual_seed(1)
    if s.op == "k2k":
        # (person, course) pairs of the graph, half of them with a near neighbour's course
        t, o = s.ctx.table(persons), s.ctx.table()
        s.ctx.known_to_unknown(t, 0, v["p_takes"], wk.OUT, o)
        pc = s.device_table(o.h).to(torch.int64)
        torch.cuda.synchronize()
        t.free(), o.free()
        at = torch.randint(0, len(pc), (R,), generator=g, device="cuda")
        half = torch.rand(R, generator=g, device="cuda") < 0.5
        rows[:, 0] = pc[at, 0]
        rows[:, cols - 1] = torch.where(half, pc[at, 1], pc[(at + 7) % len(pc), 1])
        s.args = (0, cols - 1, v["p_takes"], wk.OUT)
    else:
        rows[:, cols - 1] = p[torch.randint(0, len(p), (R,), generator=g, device="cuda")]
        s.args = {"k2u": (cols - 1, v["p_takes"], wk.OUT),
                  "k2c": (cols - 1, v["t_person_a"], wk.TYPE_ID, wk.OUT),
                  "kuu": (cols - 1, wk.OUT)}[s.op]
    s.tin = s.ctx.table(rows.to(torch.int32).cpu().numpy().view(np.uint32))
    s.tout = s.ctx.table()
    s.tables = [s.tin, s.tout]
    s.fn = {"k2u": s.ctx.known_to_unknown, "k2k": s.ctx.known_to_known, "k2c": s.ctx.known_to_const,
            "kuu": s.ctx.known_unknown_unknown}[s.op]


def _prepare_final(s, case, rng, seed):
    R, cols = case["rows"], case["cols"]
    # ids of the graph's classes, column by column: a few organisations, then units, persons,
    # courses and documents
    first, span = s.v["first_vid"], s.v["next_vid"] - s.v["first_vid"]
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    rows = torch.empty((R, cols), dtype=torch.int64, device="cuda")
    for c in range(cols):
        rows[:, c] = first + torch.randint(0, max(case["orgs"], span >> (3 * (cols - 1 - c))), (R,), generator=g,
                                           device="cuda")
    s.triples = None
    s.tin = s.ctx.table(rows.to(torch.int32).cpu().numpy().view(np.uint32))
    s.tout = s.ctx.table()
    s.tables = [s.tin, s.tout]
    s.args = list(range(case["keep"]))


def _prepare_build(s, case, rng, seed):
    s.versatile = case["versatile"]
    t = s.triples
    units = t[:200000][t[:200000, 1] == s.v["p_sub_org_of"], 0]
    s.plan(workloads.small_chain(s.v, int(units[rng.integers(len(units))])))
    s.pinned(1 << 20)
    s.triples = torch.from_numpy(t.view(np.int32)).pin_memory().numpy().view(np.uint32)


def _prepare_serve(s, case, rng, seed):
    s.build()
    s.n = case["n"]
    qs = _light(s, s.n)
    heavy = [workloads.heavy_star(s.v), workloads.heavy_triangle(s.v)]
    for k, i in enumerate(rng.permutation(case["n"])[:int(round(case["n"] * case["heavy"]))]):
        qs[i] = heavy[k % 2]
    qs = [qs[i] for i in np.random.default_rng(seed).permutation(s.n)]   # the order of arrival
    s.qs, s.keep = wk.queries_as_c(qs)
    s.res = (wk.QResult * s.n)()
    s.arrive = np.zeros(s.n)
    s.cfg = wk.ServeConfig()
    s.cfg.blind = 1
    s.pinned(1024)


_PREPARE = {"query": _prepare_query, "batch": _prepare_batch, "step": _prepare_step, "final": _prepare_final,
            "build": _prepare_build, "serve": _prepare_serve}


def prepare(case, seed):
    s = State(case, seed)
    _PREPARE[s.kind](s, case, np.random.default_rng(1), seed)
    s.ctx.sync()
    return s


def _host_query(s):
    s.check(s.lib.wk_query_execute_host(s.ctx.h, C.byref(s.q), s.mode, s.out_ptr, s.out.size, s.v2c, C.byref(s.cols),
                                        C.byref(s.rows)))
    return s.out[:s.rows.value * s.cols.value]


def run(s):
    lib, h = s.lib, s.ctx.h
    if s.kind == "query":
        if s.host:
            return _host_query(s)
        s.check(lib.wk_query_execute(h, C.byref(s.q), s.mode, C.byref(s.table), s.v2c, C.byref(s.cols),
                                     C.byref(s.rows)))
        return s.device_table(s.table)
    if s.kind == "batch":
        if s.stream:
            rc = lib.wk_batch_execute_stream(h, s.qs, s.n, s.stream, s.out_ptr, s.out.size, s.res)
        else:
            rc = lib.wk_batch_execute(h, s.qs, s.n, s.out_ptr, s.out.size, s.res)
        s.check(rc)
        r = np.frombuffer(s.res, RESULT)
        end = int(r["elem_offset"][-1]) + int(r["rows"][-1]) * int(r["cols"][-1])
        return [s.out[:end], r["rows"].view(np.int64), r["elem_offset"].view(np.int64), r["cols"], r["status"]]
    if s.kind == "step":
        s.fn(s.tin, *s.args, s.tout)
        return s.device_table(s.tout.h)
    if s.kind == "final":
        s.tin.final_process(s.args, distinct=True, out=s.tout)
        return s.device_table(s.tout.h)
    if s.kind == "build":
        s.ctx.build_store(s.triples, versatile=s.versatile)
        return _host_query(s)
    s.check(lib.wk_serve_run_open_loop(h, C.byref(s.cfg), s.qs, s.n, s.arrive.ctypes.data, s.out_ptr, s.out.size,
                                       s.res))
    r = np.frombuffer(s.res, RESULT)
    return [r["rows"].view(np.int64), r["cols"], r["status"]]


def exact(case, seed):
    return None


def _heavy_bytes(query, n):
    if query == "star":      # index, unit of each person, courses of each person; (person, unit, course) rows
        return n * (PERSONS_A * (4 + 4 + 4 * TAKES) + PERSONS_A * TAKES * 12)
    # index, unit and degree of each person, organisation of each unit; one row in n closes
    return n * (PERSONS * (4 + 4 + 4) + UNITS * 4) + PERSONS * 12


def work(case):
    """Ids read once (4 bytes per list entry and per table value) and ids written once."""
    n, kind = case["orgs"], case["kind"]
    if kind == "query":
        if case["query"] in ("star", "triangle"):
            b = _heavy_bytes(case["query"], n)
        else:     # 45 persons of a unit, their courses and the courses' types
            b = 45 * 4 + 45 * TAKES * (4 + 4 + 8)
    elif kind == "batch":    # about 375 ids of lists and 375 of tables a light query
        b = case["n"] * (80 + 3000)
    elif kind == "step":
        r, c = case["rows"], case["cols"]
        b = r * c * 4
        if case["op"] == "k2u":
            b += r * TAKES * (4 + (c + 1) * 4)
        elif case["op"] == "kuu":
            b += r * (TAKES + 6) * (4 + (c + 2) * 4)
        else:
            b += r * (4 + c * 4 * (0.6 if case["op"] == "k2k" else 0.33))
    elif kind == "final":
        b = case["rows"] * 4 * (case["cols"] + 0.5 * case["keep"])
    elif kind == "build":
        b = n * TRIPLES * (12 + STORE_BYTES)
    else:
        b = case["n"] * (80 + 1500 + case["heavy"] * 0.5 * (_heavy_bytes("star", n) + _heavy_bytes("triangle", n)))
    return {"bytes": float(b), "flops": 0.0}
