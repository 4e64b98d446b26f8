"""Benchmark of the B200 triple-pattern exploration step.

Graph: the seeded LUBM-shaped synthetic graph resident in HBM (default 10,000 organisations:
1.37e8 triples, 2.7e8 directed edges; the stated per-organisation shape gives about 13,700
triples per organisation, so this is the graph size the batching, heavy and serving workloads
are quoted on).

Headline (`value`): light-query QPS of the batched path.  One step = one batch of 16,384 light
queries (2-6 patterns from uniformly random constants of randomly drawn start classes),
all executed to their final tables by the per-level persistent launches replayed from a CUDA
graph; timed with CUDA events on the library's stream, L2 flushed between steps outside the
timed brackets.  Every query of a batch completes when the batch does, so the batch time is
each query's device latency; p50/p99 are over the timed batches.
`e2e`: light queries from host memory through wk_batch_execute_stream, 8 batches of 16,384
per call: plans in, every query's final table copied to pinned host memory, host clock
(`single_batch_call`: one batch per wk_batch_execute call).
`plain_path`: one launch per pattern per query with a host sync per step (the reference's
shape) on a sample of the same queries.
`heavy`: the heavy-query configuration's two queries (PersonA star, memberOf / subOrgOf /
degreeFrom triangle), device-resident graph replays.
`serving`: open-loop Poisson sweep of the 98 % light / 2 % heavy mix through
wk_serve_run_open_loop (continuous batching), p50/p99/p99.9 per class.
`--impl reference` times the reference's own CPU engine (oracle/_ref/libwkref.so:
sparql.hpp compiled unmodified, over the GStore arrays of the oracle's store) on all host cores
on the same light batch, one engine per thread taking whole queries, as a server's engine
threads run light queries; where that library was not built, the oracle's restatement of it.
"""
import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(ROOT, "wukong-cube_b200"))
sys.path.insert(0, os.path.join(ROOT, "oracle"))
sys.path.insert(0, os.path.join(ROOT, "oracle", "refpin"))

import numpy as np  # noqa: E402

METRIC = "light-query QPS at p99 latency; heavy-query ms; vs plain per-query GPU path"

# DRAM bytes (read + write) per input row of the dominant batch level, from one ncu capture
# (dram__bytes_read.sum + dram__bytes_write.sum) of the third fused level of a 16,384-query batch
# on the 2,000-organisation graph: 37,519,400 B + 2,610,688 B for 1,405,738 input rows.  Scaled by
# the dominant level's input rows; on the larger graph fewer sectors hit in L2, so the scaled
# figure is a lower bound there.
LEVEL_TRAFFIC_PER_ROW = (37519400 + 2610688) / 1405738
# DRAM bytes (read + write) per input row of the heavy triangle's steps run one per launch, from
# one ncu capture (dram__bytes_read.sum + dram__bytes_write.sum) on the 2,000-organisation graph
# (4.2 GB store, 1,806,383 input rows per step): the known_to_known step (degreeFrom) and the
# one-to-one known_to_unknown step (memberOf).  Scaled by the dominant heavy step's input rows.
HEAVY_TRAFFIC_PER_ROW = {
    "known_to_known": (31024640 + 512) / 1806383,
    "known_to_unknown": (16579072 + 2304) / 1806383,
}


def dram_rate(traffic_bytes, ms, peak_gbs):
    """DRAM bytes actually moved (the ncu-derived traffic) per second of the launch, beside the
    algorithmic-byte rate: a random probe moves a whole DRAM line for its 16 algorithmic bytes,
    so this is the rate at which the memory itself is kept busy."""
    gbs = traffic_bytes / (ms / 1000.0) / 1e9
    return {"gbs": gbs, "frac_of_peak": gbs / peak_gbs}


def call_latency(seconds):
    """p50 / p99 / max of host-clock call durations, in ms: every query of a call has its result
    on the host when the call returns, so this is its host-visible latency (plans in, tables
    out, copies included)."""
    ms = sorted(t * 1000.0 for t in seconds)
    return {"p50": ms[len(ms) // 2], "p99": ms[min(len(ms) - 1, int(0.99 * len(ms)))], "max": ms[-1],
            "calls": len(ms)}


def peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        d = json.load(open(p))
        return float(d["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


class Clocks:
    """Samples nvidia-smi clocks and throttle reasons while the timed region runs."""

    def __init__(self, index):
        self.index = index
        self.rows = []
        self.proc = None

    def __enter__(self):
        q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), "--query-gpu=" + q,
                                          "--format=csv,noheader,nounits", "-lms", "50"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
            time.sleep(0.3)
        except OSError:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.rows.append([x.strip() for x in line.split(",")])

    def __exit__(self, *a):
        if self.proc:
            time.sleep(0.1)
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        def num(x):
            try:
                return float(x)
            except ValueError:
                return None
        good = [r for r in self.rows if len(r) >= 9]
        if not good:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"], "samples": 0}
        sm = [num(r[1]) for r in good if num(r[1]) is not None]
        mx = [num(r[2]) for r in good if num(r[2]) is not None]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = set()
        for r in good:
            for i, n in enumerate(names):
                if r[5 + i].lower().startswith("active"):
                    reasons.add(n)
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(mx) if mx else None, "reasons": sorted(reasons),
                "samples": len(good)}


def build_graph(args):
    import wukong_b200 as wk
    t0 = time.time()
    tr, v = wk.synth_generate(args.orgs, seed=args.seed, zipf=args.zipf, zipf_s=args.zipf_s)
    t1 = time.time()
    g = wk.GStore(tr, load_factor=args.load_factor)
    t2 = time.time()
    inst = {t: g.get_index(t, wk.IN) for t in range(v["t_org"], v["t_doc"] + 1)}
    return tr, v, g, inst, {"triples": int(tr.shape[0]), "gen_s": round(t1 - t0, 2),
                            "build_s": round(t2 - t1, 2), **g.info()}


def graph_name(args):
    skew = (", degreeFrom targets and course choices Zipf s=%g" % args.zipf_s) if args.zipf else ""
    return "seeded LUBM-shaped graph of %d organisations%s" % (args.orgs, skew)


def config(args):
    """The workload, the same in both arms (graph sizes and build times go in "graph")."""
    return {"workload": "batches of %d light queries (2-6 patterns from random constants) on the "
                        "%s; heavy star + triangle alongside" % (args.light, graph_name(args)),
            "orgs": args.orgs, "seed": args.seed, "zipf": args.zipf_s if args.zipf else None,
            "light_queries_per_step": args.light,
            "l2": "flushed between timed steps (256 MiB write)"}


class CpuEngine:
    """The CPU engine the baselines time: the reference's own engine over the oracle store's
    arrays where oracle/_ref/libwkref.so exists ("reference"), else the oracle's restatement
    ("port")."""

    def __init__(self, o):
        import refengine
        self.o = o
        self.kind = "reference" if refengine.available() else "port"
        self.g = refengine.RefGraph(o) if self.kind == "reference" else None
        self.how = ("the reference's SPARQLEngine (sparql.hpp compiled unmodified) over the "
                    "oracle's GStore arrays" if self.g else
                    "the oracle (the reference CPU engine restated)")

    def run_many(self, flat, nv, threads):
        return (self.g or self.o).run_many(flat, nv, threads)

    def run_heavy(self, q, cores):
        """Status of one heavy query split into `cores` slices of its index start."""
        if self.g:
            return self.g.run_split(q.flat(), q.nvars, cores)[0]
        return self.o.run(q.flat(), q.nvars, mt_factor=cores)[0]


def run_reference(args, world, rank):
    """CPU arm: the reference's CPU engine on all host cores (CpuEngine).  The process loads the
    generator's own library (libwk_synth.so), the oracle and the reference engine, not the
    product library: the graph comes from the generator, the store and the type instances from
    the oracle."""
    if rank != 0:
        return
    import oracle
    import workloads
    import wukong_b200 as wk
    cores = os.cpu_count() or 1
    t0 = time.time()
    tr, v = wk.synth_generate(args.orgs, seed=args.seed, zipf=args.zipf, zipf_s=args.zipf_s,
                              generator_only=True)
    t1 = time.time()
    o = oracle.OracleStore(tr)
    t2 = time.time()
    inst = {t: o.get_index(t, wk.IN) for t in range(v["t_org"], v["t_doc"] + 1)}
    ginfo = {"triples": int(tr.shape[0]), "gen_s": round(t1 - t0, 2), "build_s": round(t2 - t1, 2),
             "store": "oracle"}
    qs = workloads.light_queries(v, inst, args.light, seed=args.seed + 1)
    flat = [q.flat() for q in qs]
    nv = [q.nvars for q in qs]
    eng = CpuEngine(o)
    for _ in range(args.warmup):
        eng.run_many(flat, nv, cores)
    times = []
    for _ in range(args.steps):
        t0 = time.perf_counter()
        _, st = eng.run_many(flat, nv, cores)
        times.append(time.perf_counter() - t0)
        assert (st == 0).all()
    value = len(qs) * args.steps / sum(times)
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": "light queries/s",
            "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": 1000 * sum(times) / len(times), "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "u32", "data": "synthetic",
            "config": config(args), "graph": ginfo,
            "cpu_baseline": {"value": value, "unit": "light queries/s", "cores": cores, "kind": eng.kind,
                             "sample": "%d steps x %d light queries after %d warm-up steps, one "
                                       "query per thread; %s" % (args.steps, len(qs), args.warmup, eng.how)},
            "e2e": {"value": value, "unit": "light queries/s", "h2d_bytes_per_step": 0,
                    "d2h_bytes_per_step": 0}}
    print(json.dumps(line))


def timed(stream, flush, steps, fn):
    """Per-step device ms with CUDA events on `stream`; L2 flushed outside the brackets."""
    import torch
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
          for _ in range(steps)]
    torch.cuda.synchronize()
    for i in range(steps):
        with torch.cuda.stream(stream):
            flush.zero_()
            ev[i][0].record(stream)
        fn()
        with torch.cuda.stream(stream):
            ev[i][1].record(stream)
    torch.cuda.synchronize()
    return [a.elapsed_time(b) for a, b in ev]


def _pct(x, p):
    return float(np.percentile(x, p)) if len(x) else None


def serving_sweep(ctx, v, inst, o, args, plain_qps, heavy_rows):
    """Open-loop Poisson arrivals at each offered rate: 98 % light queries (the batch shapes),
    2 % heavy ones (star and triangle alternating), replies blind (row counts only, as the
    reference's emulator runs).  Light and heavy latency percentiles are arrival -> reply on the
    host clock; `sustained` is the highest offered rate whose light p99 stays within 1 ms while
    completions keep up with arrivals."""
    import workloads
    hq = [workloads.heavy_star(v), workloads.heavy_triangle(v)]
    # warm-up run (untimed): loads every kernel of the serving path and builds the lanes
    wq = workloads.light_queries(v, inst, 1000, seed=args.seed + 4999)
    wq[::50] = [hq[j % 2] for j in range(len(wq[::50]))]
    ctx.serve(wq, np.linspace(0, 50000, len(wq)), blind=1, max_heavy_inflight=args.serve_lanes,
              light_ctas_per_sm=args.serve_light_ctas)
    sweep = []
    for k, qps in enumerate(args.serve_rates):
        rng = np.random.default_rng(args.seed + 7000 + k)
        n = int(max(500, qps * args.serve_seconds))
        qs = workloads.light_queries(v, inst, n, seed=args.seed + 5000 + k)
        is_heavy = np.zeros(n, bool)
        hidx = rng.choice(n, size=max(1, n // 50), replace=False)
        for j, i in enumerate(hidx):
            qs[i] = hq[j % 2]
            is_heavy[i] = True
        arrivals = np.cumsum(rng.exponential(1e6 / qps, size=n))
        res = ctx.serve(qs, arrivals, blind=1, max_heavy_inflight=args.serve_lanes,
                        light_ctas_per_sm=args.serve_light_ctas)
        st = np.array([r[1] for r in res])
        rows = np.array([r[4] for r in res], np.int64)
        lat = np.array([r[3] - r[2] for r in res])
        assert (st == 0).all(), "serving: a query failed"
        if o is not None and not args.no_check:
            light = np.nonzero(~is_heavy)[0]
            orows, ost = o.run_many([qs[i].flat() for i in light], [qs[i].nvars for i in light],
                                    os.cpu_count() or 1)
            assert np.array_equal(orows.astype(np.int64), rows[light]), "serving row counts differ"
            for j, i in enumerate(hidx):
                assert rows[i] == heavy_rows[j % 2], "serving heavy row count differs"
        done = np.array([r[3] for r in res])
        span = (done.max() - arrivals[0]) / 1e6
        light_span = (done[~is_heavy].max() - arrivals[0]) / 1e6
        heavy_span = (done[is_heavy].max() - arrivals[0]) / 1e6
        ll, hl = lat[~is_heavy], lat[is_heavy]
        sweep.append({"offered_qps": qps, "queries": n, "heavy": int(is_heavy.sum()),
                      "completed_qps": n / span,
                      "light_completed_qps": int((~is_heavy).sum()) / light_span,
                      "light_offered_qps": qps * float((~is_heavy).mean()),
                      "heavy_completed_qps": int(is_heavy.sum()) / heavy_span,
                      "heavy_offered_qps": qps * float(is_heavy.mean()),
                      "light_us": {"p50": _pct(ll, 50), "p99": _pct(ll, 99), "p99.9": _pct(ll, 99.9)},
                      "heavy_us": {"p50": _pct(hl, 50), "p99": _pct(hl, 99), "max": float(hl.max())}})
    # light-only: the highest offered rate whose light p99 stays within 1 ms while light
    # completions keep up with light arrivals.  Both classes: the highest offered rate where,
    # in addition, heavy completions keep up with heavy arrivals and the heavy p99 stays
    # within 5 ms.
    ok = [s for s in sweep if s["light_us"]["p99"] <= 1000.0 and
          s["light_completed_qps"] >= 0.95 * s["light_offered_qps"]]
    best = max(ok, key=lambda s: s["offered_qps"]) if ok else None
    both = [s for s in ok if s["heavy_us"]["p99"] <= 5000.0 and
            s["heavy_completed_qps"] >= 0.95 * s["heavy_offered_qps"]]
    best2 = max(both, key=lambda s: s["offered_qps"]) if both else None
    return {"mix": ("98% light (batch shapes) / 2% heavy (star, triangle); open-loop Poisson; "
                    "blind replies (row counts); heavy queries on {} low-priority lanes; admission "
                    "by each query's projected bytes").format(args.serve_lanes),
            "sweep": sweep,
            "sustained_qps_light_p99_le_1ms": best["light_offered_qps"] if best else None,
            "sustained_offered_qps_at_that_point": best["offered_qps"] if best else None,
            "sustained_vs_plain": (best["light_offered_qps"] / plain_qps) if best else None,
            "sustained_offered_qps_both_classes": best2["offered_qps"] if best2 else None,
            "both_classes_rule": "light p99 <= 1 ms, heavy p99 <= 5 ms, each class completing "
                                 ">= 95% of its offered rate"}


def distinct_probe_keys(ctx, q, k):
    """Distinct keys step k of query q probes: 1 for the start (one index or constant key),
    else the distinct values of the step's known subject column in the table of the first k
    patterns (run on the device; its tables match the oracle's)."""
    import wukong_b200 as wk
    if k == 0:
        return 1
    s = q.patterns[k][0]
    prefix = wk.Query(q.patterns[:k], nvars=q.nvars)
    table, v2c = ctx.execute(prefix, wk.MODE_RESIDENT)
    return int(np.unique(table[:, v2c[-s - 1]]).size)


def run_ours(args, world, rank, local_rank):
    import torch

    import oracle
    import replicas
    import workloads
    import wukong_b200 as wk

    torch.cuda.set_device(local_rank)
    tr, v, g, inst, ginfo = build_graph(args)
    ctx = wk.Context(local_rank)
    ctx.upload_gstore(g)
    ginfo["device_store_bytes"] = ctx.store_bytes()
    if not args.no_device_build:
        # the same store built on the device (wk_store_build_device) from the same triples, in a
        # second context: wall time of the call (upload of the triples included), against the
        # host build above; the two stores must hold the same slots and lists
        with wk.Context(local_rank) as cb:
            cb.build_store(tr[:1], load_factor=args.load_factor)   # loads the build's kernels
            t0 = time.time()
            cb.build_store(tr, load_factor=args.load_factor)
            ginfo["device_build_s"] = round(time.time() - t0, 3)
            same = cb.store_bytes() == ginfo["device_store_bytes"]
            probe = workloads.light_queries(v, inst, 512, seed=args.seed + 3)
            a = [r[0].shape[0] if r[0] is not None else -1 for r in cb.batch(probe)]
            b = [r[0].shape[0] if r[0] is not None else -1 for r in ctx.batch(probe)]
            assert same and a == b, "device-built store differs from the host-built one"
    stream = torch.cuda.ExternalStream(ctx.stream())
    flush = torch.empty(64 << 20, dtype=torch.int32, device="cuda")
    cores = os.cpu_count() or 1
    o = oracle.OracleStore(tr) if rank == 0 else None
    eng = CpuEngine(o) if o is not None else None

    # ---- light batch: correctness gate, then timing.  With N GPUs (replicas) the query stream
    # holds N batches and each rank answers its own share of it.
    stream_qs = workloads.light_queries(v, inst, args.light * world, seed=args.seed + 1)
    lo, hi = replicas.shard(len(stream_qs), rank, world)
    qs = stream_qs[lo:hi]
    res = ctx.batch(qs)
    light_rows = np.array([r[0].shape[0] if r[0] is not None else 0 for r in res], np.int64)
    if o is not None and not args.no_check:
        orows, ost = o.run_many([q.flat() for q in qs], [q.nvars for q in qs], cores)
        assert (ost == 0).all() and np.array_equal(orows.astype(np.int64), light_rows), \
            "light batch row counts differ from the oracle"
        for i in range(0, len(qs), max(1, len(qs) // 256)):
            st, want, _ = o.run(qs[i].flat(), qs[i].nvars)
            assert np.array_equal(oracle.sorted_rows(res[i][0]), oracle.sorted_rows(want)), i
    # the autotuner picks the tile schedule (lanes, slice threshold) on this batch and on the
    # heavy queries; the timed runs below use its choice
    tune = ctx.autotune(qs + [workloads.heavy_star(v), workloads.heavy_triangle(v)], iters=3)
    ctx.batch_device(qs)   # capture for replay
    for _ in range(args.warmup):
        ctx.batch_replay()
    ctx.check()
    if world > 1:
        torch.distributed.barrier()
    with Clocks(local_rank) as clk:
        # the light-batch timed region as an NVTX range, so an ncu launch list can pick it
        # (ncu --nvtx --nvtx-include "timed/")
        torch.cuda.nvtx.range_push("timed")
        step_ms = timed(stream, flush, args.steps, ctx.batch_replay)
        torch.cuda.nvtx.range_pop()
    ctx.check()
    tot_ms = replicas.max_over_ranks(sum(step_ms), device="cuda")   # whole-job device time
    value = replicas.sum_over_ranks(len(qs), device="cuda") * args.steps / (tot_ms / 1000.0)

    # ---- e2e through the C ABI from the host (plans in, tables out to pinned memory)
    qs_c, keep = wk.queries_as_c(qs)
    total_elems = int(sum((r[0].size if r[0] is not None else 0) for r in res))
    host = torch.empty(total_elems + 1024, dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)
    qres = (wk.QResult * len(qs))()
    import ctypes as C
    L = wk.lib()
    rc = L.wk_batch_execute(ctx.h, qs_c, len(qs), C.c_void_p(host.ctypes.data), host.size, qres)
    assert rc == 0
    one_t = []
    for _ in range(args.steps):
        t0 = time.perf_counter()
        rc = L.wk_batch_execute(ctx.h, qs_c, len(qs), C.c_void_p(host.ctypes.data), host.size, qres)
        one_t.append(time.perf_counter() - t0)
        assert rc == 0
    e2e_single = len(qs) * args.steps / sum(one_t)

    # the headline end-to-end number: a stream of e2e_batches batches per call through
    # wk_batch_execute_stream (plans resolved on the host, descriptors uploaded, every table
    # copied back to pinned host memory, batch i's copy and batch i+1's plans overlapping the
    # device work), wall clock around each call
    e2e_qs = workloads.light_queries(v, inst, args.light * args.e2e_batches, seed=args.seed + 77 + rank)
    eq_c, keep_e = wk.queries_as_c(e2e_qs)
    eres = (wk.QResult * len(e2e_qs))()
    ecap = int(total_elems * args.e2e_batches * 1.5) + (1 << 20)
    ehost = torch.empty(ecap, dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)
    rc = L.wk_batch_execute_stream(ctx.h, eq_c, len(e2e_qs), args.light, C.c_void_p(ehost.ctypes.data),
                                   ehost.size, eres)
    assert rc == 0, wk.lib().wk_last_error(ctx.h)
    erows = np.array([eres[i].rows for i in range(len(e2e_qs))], np.int64)
    if o is not None and not args.no_check:
        orows, ost = o.run_many([q.flat() for q in e2e_qs], [q.nvars for q in e2e_qs], cores)
        assert (ost == 0).all() and np.array_equal(orows.astype(np.int64), erows), \
            "streamed batch row counts differ from the oracle"
    e2e_t = []
    for _ in range(args.steps):
        t0 = time.perf_counter()
        rc = L.wk_batch_execute_stream(ctx.h, eq_c, len(e2e_qs), args.light,
                                       C.c_void_p(ehost.ctypes.data), ehost.size, eres)
        e2e_t.append(time.perf_counter() - t0)
        assert rc == 0
    e2e = len(e2e_qs) * args.steps / sum(e2e_t)
    e_elems = int(sum(eres[i].rows * eres[i].cols for i in range(len(e2e_qs))))
    h2d = 0
    for s in range(0, len(e2e_qs), args.light):   # descriptors of every level, steps, widths
        part = e2e_qs[s:s + args.light]
        h2d += max(len(q.patterns) for q in part) * len(part) * 64 + len(part) * 8
    d2h = e_elems * 4 + len(e2e_qs) * 16

    # ---- plain path (one launch per pattern, host sync per step) and the single-query
    # resident path on a sample of the same queries
    sample = qs[:args.plain_sample]
    buf = np.zeros(max(int(light_rows.max()) * 8, 64), np.uint32)
    for q in sample[:8]:
        ctx.execute_host(q, buf, wk.MODE_PLAIN)
    t0 = time.perf_counter()
    for q in sample:
        ctx.execute_host(q, buf, wk.MODE_PLAIN)
    plain = len(sample) / (time.perf_counter() - t0)
    t0 = time.perf_counter()
    for q in sample:
        ctx.execute_host(q, buf, wk.MODE_RESIDENT)
    single_resident = len(sample) / (time.perf_counter() - t0)

    # ---- heavy queries (device-resident graph replays)
    hq = [workloads.heavy_star(v), workloads.heavy_triangle(v)]
    heavy_rows = []
    heavy_cpu = {}
    for name, q in zip(("star", "triangle"), hq):
        got, _ = ctx.execute(q, wk.MODE_GRAPH)
        heavy_rows.append(int(got.shape[0]))
        if o is not None and not args.no_check:
            st, want, _ = o.run(q.flat(), q.nvars, mt_factor=cores)
            assert st == 0 and np.array_equal(oracle.sorted_rows(got), oracle.sorted_rows(want))
        if o is not None and not args.no_cpu:
            # the CPU engine on every host core, split as the reference splits an index start
            # (mt_factor slices of the index list, one per thread; sparql.hpp:213-224), after
            # one warm run
            eng.run_heavy(q, cores)
            cpu_t = []
            for _ in range(args.heavy_cpu_reps):
                t0 = time.perf_counter()
                st = eng.run_heavy(q, cores)
                cpu_t.append((time.perf_counter() - t0) * 1000)
                assert st == 0
            heavy_cpu[name] = statistics.median(cpu_t) if cpu_t else None
    heavy = {}
    for name, q in zip(("star", "triangle"), hq):
        ms = timed(stream, flush, args.steps, lambda q=q: ctx.enqueue(q, wk.MODE_GRAPH))
        ctx.check()
        t0 = time.perf_counter()
        for _ in range(3):
            ctx.execute(q, wk.MODE_PLAIN)
        plain_ms = (time.perf_counter() - t0) / 3 * 1000
        heavy[name] = {"ms": statistics.median(ms), "rows": heavy_rows[len(heavy)],
                       "plain_ms": plain_ms, "profile": ctx.profile(q, iters=3),
                       "cpu_ms": heavy_cpu.get(name), "cpu_cores": cores,
                       "cpu_how": "%s, mt_factor = cores, median of %d runs after a warm run"
                                  % (eng.how if eng else "", args.heavy_cpu_reps)}
        if heavy_cpu.get(name):
            heavy[name]["speedup_vs_cpu"] = heavy_cpu[name] / heavy[name]["ms"]

    # ---- post-pattern stage on the device: DISTINCT ?x2 ?x1 over the heavy star's table, as the
    # star leaves it (already in the sort's order, so the sort is skipped) and with its rows
    # shuffled (the radix sort runs); the sort's order is canonical, so both give the same rows
    star_table, star_v2c = ctx.execute(hq[0], wk.MODE_RESIDENT)
    keep = [star_v2c[1], star_v2c[0]]

    def time_distinct(table):
        pin = wk.Table(ctx, max(table.size, 1))
        pin.upload(table)
        pout = pin.final_process(keep, distinct=True)   # warm: the output table and scratch grow once
        ms = []
        for _ in range(5):
            t0 = time.perf_counter()
            pin.final_process(keep, distinct=True, out=pout)
            ms.append((time.perf_counter() - t0) * 1000)
        rows = pout.download()
        pout.free()
        pin.free()
        return statistics.median(ms), rows

    pp_ms, pp_out = time_distinct(star_table)
    shuffled = star_table[np.random.default_rng(args.seed).permutation(star_table.shape[0])]
    pp_sh_ms, pp_sh_out = time_distinct(shuffled)
    assert np.array_equal(pp_out, pp_sh_out), "DISTINCT differs on the shuffled rows"
    del shuffled, pp_sh_out
    post_pattern = {"op": "DISTINCT on two of the heavy star's three columns (wk_table_final_process)",
                    "rows_in": int(star_table.shape[0]), "cols_in": int(star_table.shape[1]),
                    "rows_out": int(pp_out.shape[0]), "ms": pp_ms,
                    "ms_rows_shuffled": pp_sh_ms,
                    "timing": "host clock around the call (it ends with a device sync), median of 5 "
                              "after a warm call, output table reused; ms: the table as the star "
                              "leaves it (in the sort's order: the sort is skipped), "
                              "ms_rows_shuffled: the same rows shuffled (radix sort), same result"}

    # ---- serving: open-loop Poisson sweep, 98 % light / 2 % heavy, blind replies
    serving = None
    if not args.no_serve:
        serving = serving_sweep(ctx, v, inst, o, args, plain, heavy_rows)

    # ---- roofline: dominant kernel of the light batch (one level launch), CUDA events on the
    # library stream; and of the heavy queries
    peak, src = peaks()
    prof = ctx.batch_profile(qs, iters=3)
    levels = [s for s in prof if s["kind"] == "batch_level"]
    overheads = {s["kind"]: s["ms"] for s in prof if s["kind"] != "batch_level"}
    dom = max(levels, key=lambda s: s["ms"])
    achieved = dom["alg_bytes"] / (dom["ms"] / 1000.0) / 1e9
    hsteps = [s for h in heavy.values() for s in h["profile"]]
    hdom = max(hsteps, key=lambda s: s["ms"])
    hach = hdom["alg_bytes"] / (hdom["ms"] / 1000.0) / 1e9
    # the random-read ceiling of this GPU, measured here: a probe is a random 16-byte read, and
    # on this part each one moves a whole 128-byte line from DRAM, so the copy bandwidth
    # overstates what probes can reach
    rr_peak = ctx.measure_random_reads(8 << 30, iters=5)

    def bound_s(s):
        # a lower bound on a step's time: one random read per distinct probed key (its bucket
        # must come from DRAM at least once; the store is far larger than L2) at the measured
        # random-read rate, or its algorithmic bytes at the copy bandwidth, whichever is longer
        return max(s["distinct_keys"] / rr_peak, s["alg_bytes"] / (peak * 1e9))

    def random_roofline(s):
        return {"bound": "hash probes: one random read per distinct probed key at the measured random-read "
                         "rate, or the algorithmic bytes at the copy bandwidth, whichever is longer "
                         "(lookups by vertex directory share lines between keys and may pass it)",
                "distinct_keys": s["distinct_keys"], "peak_reads_per_s": rr_peak,
                "peak_bytes_per_s": peak * 1e9, "bound_ms": bound_s(s) * 1000.0,
                "kernel_ms": s["ms"], "frac": bound_s(s) / (s["ms"] / 1000.0)}
    for q, h in zip(hq, heavy.values()):
        for k, s in enumerate(h["profile"]):
            s["distinct_keys"] = distinct_probe_keys(ctx, q, k)
        h["bound_ms"] = sum(bound_s(s) for s in h["profile"]) * 1000.0
        h["frac_of_bound"] = h["bound_ms"] / sum(s["ms"] for s in h["profile"])
    flat_mask = tune.get("batch_flat", 0)
    dom_k = levels.index(dom)
    dom_kernel = ("level_kernel (fused batch level %d)" if not flat_mask else
                  "flat passes (batch level %d)" if (flat_mask >> dom_k) & 1
                  else "explore_kernel (batch level %d)") % dom_k

    lat = sorted(step_ms)
    line = {"metric": METRIC, "value": value, "unit": "light queries/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": tot_ms / args.steps,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u32",
            "data": "synthetic", "config": config(args), "graph": ginfo,
            "latency_ms": {"p50": lat[len(lat) // 2], "p99": lat[min(len(lat) - 1, int(0.99 * len(lat)))],
                           "max": lat[-1], "note": "every query of a batch completes with the batch"},
            "e2e": {"value": e2e, "unit": "light queries/s", "h2d_bytes_per_step": h2d,
                    "d2h_bytes_per_step": d2h,
                    "step": "one wk_batch_execute_stream call: %d batches of %d light queries"
                            % (args.e2e_batches, args.light),
                    "latency_ms_per_call": call_latency(e2e_t),
                    "single_batch_call": {"value": e2e_single, "unit": "light queries/s",
                                          "api": "wk_batch_execute, one batch per call",
                                          "latency_ms_per_call": call_latency(one_t)}},
            "plain_path": {"value": plain, "unit": "light queries/s", "sample": len(sample)},
            "single_query_resident": {"value": single_resident, "unit": "light queries/s"},
            "speedup_vs_plain": value / plain,
            "light_rows": {"p50": int(np.percentile(light_rows, 50)),
                           "p99": int(np.percentile(light_rows, 99)), "max": int(light_rows.max())},
            "heavy": heavy,
            "post_pattern": post_pattern,
            "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                         "frac": achieved / peak, "traffic": LEVEL_TRAFFIC_PER_ROW * dom["rows_in"],
                         "traffic_rate": dram_rate(LEVEL_TRAFFIC_PER_ROW * dom["rows_in"], dom["ms"], peak),
                         "traffic_source": "ncu dram__bytes_read.sum + dram__bytes_write.sum of "
                                           "the third fused level on the 2,000-organisation graph "
                                           "(28.5 B per input row) x this launch's input rows",
                         "peak_source": src,
                         "kernel": dom_kernel,
                         "algorithmic_bytes": dom["alg_bytes"], "kernel_ms": dom["ms"],
                         "probe_rate": {"probes_per_s": dom["rows_in"] / (dom["ms"] / 1000.0),
                                        "frac_of_random_read_peak":
                                            dom["rows_in"] / (dom["ms"] / 1000.0) / rr_peak,
                                        "note": "one probe per input row"}},
            "roofline_heavy": {"bound": "hbm", "achieved": hach, "peak": peak, "unit": "GB/s",
                               "frac": hach / peak,
                               "traffic": (HEAVY_TRAFFIC_PER_ROW[hdom["kind"]] * hdom["rows_in"]
                                           if hdom["kind"] in HEAVY_TRAFFIC_PER_ROW else None),
                               "traffic_rate": (dram_rate(HEAVY_TRAFFIC_PER_ROW[hdom["kind"]] * hdom["rows_in"],
                                                          hdom["ms"], peak)
                                                if hdom["kind"] in HEAVY_TRAFFIC_PER_ROW else None),
                               "traffic_source": "ncu dram__bytes_read.sum + dram__bytes_write.sum of "
                                                 "the triangle's steps on the 2,000-organisation "
                                                 "graph (1 pass; B per input row of this step's kind) x "
                                                 "this step's input rows",
                               "kernel": "pipe_kernel (single-query " + hdom["kind"] + " step, one per launch)",
                               "algorithmic_bytes": hdom["alg_bytes"], "kernel_ms": hdom["ms"],
                               "random_reads": random_roofline(hdom)},
            "random_read_peak": {"value": rr_peak, "unit": "reads/s",
                                 "how": "wk_measure_random_reads: independent random 16-byte "
                                        "reads from an 8 GiB device buffer, CUDA events"},
            "batch_levels": levels,
            "batch_other_ms": overheads,
            "autotune": tune,
            "serving": serving,
            # per batch: one launch per level (three where the level runs the flat passes; fused
            # levels are fewer than the patterns), result scan, gather
            "gpu_launches": args.steps * (sum(3 if (tune.get("batch_flat", 0) >> k) & 1 else 1
                                              for k in range(len(levels))) + 2),
            "clocks": clk.summary()}
    if rank == 0:
        if not args.no_cpu:
            # the reference arm's method: warm-up runs, then --steps timed runs of the same batch
            flat, nv = [q.flat() for q in qs], [q.nvars for q in qs]
            for _ in range(args.warmup):
                eng.run_many(flat, nv, cores)
            cpu_t = []
            for _ in range(args.steps):
                t0 = time.perf_counter()
                _, st = eng.run_many(flat, nv, cores)
                cpu_t.append(time.perf_counter() - t0)
                assert (st == 0).all()
            line["cpu_baseline"] = {"value": len(qs) * len(cpu_t) / sum(cpu_t), "unit": "light queries/s",
                                    "cores": cores, "kind": eng.kind,
                                    "sample": "%d steps x %d light queries after %d warm-up steps, one "
                                              "query per thread; %s" % (args.steps, len(qs), args.warmup,
                                                                        eng.how)}
        print(json.dumps(line))
    ctx.close()


def run_scale(args):
    """The scale configuration on one GPU: the store built on the device straight from the
    generator's triples (no host store), its footprint, the light batch and the heavy queries
    timed on it.  With --scale-check N the store is copied back to host memory
    (wk_store_export) and the reference's CPU engine, reading those arrays in place, answers N
    of the light queries and both heavy queries: their row counts must equal the device's."""
    import torch

    import workloads
    import wukong_b200 as wk
    t0 = time.time()
    tr, v = wk.synth_generate(args.orgs, seed=args.seed, zipf=args.zipf, zipf_s=args.zipf_s)
    gen_s = time.time() - t0
    info = {"triples": int(tr.shape[0]), "gen_s": round(gen_s, 1), "load_factor": args.load_factor or 0.1}
    ctx = wk.Context(0)
    free0, total = torch.cuda.mem_get_info()
    t0 = time.time()
    ctx.build_store(tr, load_factor=args.load_factor)
    info["device_build_s"] = round(time.time() - t0, 2)
    info["store_bytes"] = ctx.store_bytes()
    del tr
    # type instances from the device's index lists (get_index(t, IN))
    inst = {}
    t = ctx.table(capacity=1 << 20)
    for ty in range(v["t_org"], v["t_doc"] + 1):
        ctx.index_to_unknown(ty, wk.IN, t)
        inst[ty] = t.download().reshape(-1).copy()
    qs = workloads.light_queries(v, inst, args.light, seed=args.seed + 1)
    res = ctx.batch(qs)
    light_rows = np.array([r[0].shape[0] if r[0] is not None else -1 for r in res], np.int64)
    assert (light_rows >= 0).all(), "a light query failed"
    stream = torch.cuda.ExternalStream(ctx.stream())
    flush = torch.empty(64 << 20, dtype=torch.int32, device="cuda")
    ctx.batch_device(qs)
    for _ in range(args.warmup):
        ctx.batch_replay()
    ctx.check()
    with Clocks(0) as clk:
        step_ms = timed(stream, flush, args.steps, ctx.batch_replay)
    ctx.check()
    hq = {"star": workloads.heavy_star(v), "triangle": workloads.heavy_triangle(v)}
    heavy = {}
    for name, q in hq.items():
        got, _ = ctx.execute(q, wk.MODE_GRAPH)
        ms = timed(stream, flush, args.steps, lambda q=q: ctx.enqueue(q, wk.MODE_GRAPH))
        ctx.check()
        heavy[name] = {"ms": statistics.median(ms), "rows": int(got.shape[0])}
    free1, _ = torch.cuda.mem_get_info()
    info["device_used_bytes"] = int(free0 - free1)
    info["device_total_bytes"] = int(total)
    check = None
    if args.scale_check:
        import refengine
        slots, edges, segs = ctx.export_store()
        rows = np.array([[m["index"], m["pid"], m["dir"], m["num_keys"], m["num_buckets"], m["bucket_start"],
                          m["num_edges"], m["edge_start"], m["ext_start"], m["ext_num"]] for m in segs], np.uint64)
        rg = refengine.RefGraph(arrays=(slots.ctypes.data, slots.shape[0], edges.ctypes.data, rows))
        cores = os.cpu_count() or 1
        pick = list(range(0, len(qs), max(1, len(qs) // args.scale_check)))[:args.scale_check]
        rrows, rst = rg.run_many([qs[i].flat() for i in pick], [qs[i].nvars for i in pick], cores)
        assert (rst == 0).all() and np.array_equal(rrows.astype(np.int64), light_rows[pick]), \
            "light row counts differ from the reference engine"
        for name, q in hq.items():
            st, n = rg.run_split(q.flat(), q.nvars, cores)
            assert st == 0 and n == heavy[name]["rows"], name
        check = {"light_queries": len(pick), "heavy": list(hq),
                 "how": "row counts equal the reference's CPU engine reading the exported store"}
    line = {"metric": "scale configuration: light-query QPS, heavy-query ms, single-GPU footprint",
            "value": len(qs) * args.steps / (sum(step_ms) / 1000.0), "unit": "light queries/s",
            "n_gpus": 1, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": statistics.median(step_ms), "higher_is_better": True, "dtype": "u32",
            "data": "synthetic", "config": config(args), "graph": info, "heavy": heavy,
            "parity": check, "clocks": clk.summary()}
    print(json.dumps(line))
    ctx.close()


def run_profile_case(args):
    """A small, self-contained case for ncu: one heavy query (`--heavy`, resident mode) and one
    light batch, each run `--steps` times after `--warmup` runs, no oracle, no timing.  The
    batch replays after the first sit in an NVTX range named "replay", so a capture can pick
    a level of a replay (ncu --nvtx --nvtx-include replay/) whatever reruns came before."""
    import torch

    import workloads
    import wukong_b200 as wk
    tr, v, g, inst, ginfo = build_graph(args)
    with wk.Context(0) as ctx:
        ctx.upload_gstore(g)
        ctx.tune_set(wk.KNOB_BATCH_FLAT, args.batch_flat)
        if args.batch_lanes:
            ctx.tune_set(wk.KNOB_BATCH_LANES, args.batch_lanes)
        if args.batch_slice_rows:
            ctx.tune_set(wk.KNOB_BATCH_SLICE_ROWS, args.batch_slice_rows)
        q = workloads.heavy_star(v) if args.heavy == "star" else workloads.heavy_triangle(v)
        qs = workloads.light_queries(v, inst, args.light, seed=args.seed + 1)
        for _ in range(args.warmup + args.steps):
            ctx.execute(q, wk.MODE_RESIDENT)
        ctx.batch_device(qs)
        ctx.batch_replay()
        ctx.sync()
        torch.cuda.nvtx.range_push("replay")
        for _ in range(args.warmup + args.steps - 1):
            ctx.batch_replay()
        ctx.sync()
        torch.cuda.nvtx.range_pop()
        ctx.check()
    print(json.dumps({"profile_case": "ok", "graph": ginfo}))


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--profile-case", action="store_true",
                    help="run the small ncu case instead of the benchmark")
    ap.add_argument("--batch-flat", type=lambda x: int(x, 0), default=0,
                    help="profile case: mask of the batch levels run as the flat passes")
    ap.add_argument("--batch-lanes", type=int, default=0,
                    help="profile case: lanes per probe group of the batch levels (0: default)")
    ap.add_argument("--batch-slice-rows", type=int, default=0,
                    help="profile case: slice threshold of the batch levels (0: default)")
    ap.add_argument("--heavy", default="triangle", choices=["triangle", "star"],
                    help="profile case: the heavy query it runs")
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--orgs", type=int, default=10000,
                    help="organisations of the synthetic graph (10,000 give the 1.37e8-triple "
                         "graph, 2.7e8 directed edges)")
    ap.add_argument("--light", type=int, default=16384)
    ap.add_argument("--plain-sample", type=int, default=512)
    ap.add_argument("--e2e-batches", type=int, default=8,
                    help="batches per end-to-end call (wk_batch_execute_stream)")
    ap.add_argument("--seed", type=int, default=0)
    ap.add_argument("--zipf", action="store_true",
                    help="Zipf-skewed degreeFrom targets and course choices (the scale-and-skew "
                         "configuration: hub organisations and popular courses)")
    ap.add_argument("--zipf-s", type=float, default=1.1, help="Zipf exponent with --zipf")
    ap.add_argument("--load-factor", type=float, default=0.0,
                    help="store load factor (fraction of a bucket's 7 data slots in use; 0: the "
                         "builder's default 0.1)")
    ap.add_argument("--no-check", action="store_true")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-serve", action="store_true")
    ap.add_argument("--no-device-build", action="store_true",
                    help="skip timing the store build on the device against the host build")
    ap.add_argument("--heavy-cpu-reps", type=int, default=3,
                    help="timed CPU-engine runs of each heavy query (median reported)")
    ap.add_argument("--serve-rates", type=lambda s: [int(x) for x in s.split(",")],
                    default=[1000, 10000, 25000, 50000, 65000, 80000, 100000, 125000, 150000, 200000, 500000])
    ap.add_argument("--serve-seconds", type=float, default=0.25,
                    help="arrival span of each serving rate")
    ap.add_argument("--device-store", action="store_true",
                    help="the scale run: store built on the device only, footprint, light batch "
                         "and heavy queries (no host store, oracle or serving)")
    ap.add_argument("--scale-check", type=int, default=0,
                    help="with --device-store: light queries checked against the reference "
                         "engine over the exported store (needs host memory for the store)")
    ap.add_argument("--serve-lanes", type=int, default=1,
                    help="serving: index-start queries running at once, one lane each")
    ap.add_argument("--serve-light-ctas", type=int, default=0,
                    help="serving: exploration CTAs per SM of the iteration launches (0: the library's "
                         "default); the lanes' launches are sized to leave room for one more")
    args = ap.parse_args()
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    if args.profile_case:
        run_profile_case(args)
        return
    if args.device_store:
        run_scale(args)
        return
    if args.impl == "reference":
        run_reference(args, world, rank)
        return
    if world > 1:
        import datetime

        import torch
        torch.cuda.set_device(local_rank)
        torch.distributed.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))
    try:
        run_ours(args, world, rank, local_rank)
    finally:
        if world > 1:
            import torch
            torch.distributed.destroy_process_group()


if __name__ == "__main__":
    main()
