"""Vertex directories on a device that fills up: an allocation that has no other room takes theirs, and
every call answers as before, by hash; a store loaded later has directories again."""
import numpy as np
import pytest

import oracle
import workloads
import wukong_b200 as wk

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _same(got, want):
    return np.array_equal(oracle.sorted_rows(got), oracle.sorted_rows(want))


def _check(ctx, heavy, qs, o):
    for q in heavy:
        want = o.run(q.flat(), q.nvars)[1]
        for mode in (wk.MODE_PLAIN, wk.MODE_RESIDENT, wk.MODE_GRAPH):
            assert _same(ctx.execute(q, mode)[0], want)
    want = [o.run(q.flat(), q.nvars)[1] for q in qs]
    for got in (ctx.batch(qs), ctx.batch(qs, stream_batch=40)):
        assert all(st == 0 and _same(t, w) for (t, st), w in zip(got, want))
    ctx.batch_device(qs)
    ctx.batch_replay()
    ctx.check()
    mixed = qs[:20] + heavy[:1]
    for q, r in zip(mixed, ctx.serve(mixed, np.zeros(len(mixed)), arena_bytes=1 << 22)):
        assert r[1] == 0 and _same(r[0], o.run(q.flat(), q.nvars)[1])


@pytest.mark.parametrize("served", [False, True])
def test_room_of_the_directories(built, served):
    import torch
    tr, v = wk.synth_generate(150, seed=3)
    o = oracle.OracleStore(tr)
    heavy = [workloads.heavy_star(v), workloads.heavy_triangle(v)]
    with wk.Context(0, rbuf_bytes=8 * MB) as ctx:
        ctx.build_store(tr)
        inst = {}
        for t in range(v["t_org"], v["t_doc"] + 1):
            tab = ctx.table()
            ctx.index_to_unknown(t, wk.IN, tab)
            inst[t] = tab.download().reshape(-1)
            tab.free()
        qs = workloads.light_queries(v, inst, 100, seed=5)
        _check(ctx, heavy, qs, o) if served else ctx.execute(heavy[0], wk.MODE_GRAPH)
        held = torch.empty(torch.cuda.mem_get_info()[0] - 64 * MB, dtype=torch.uint8, device="cuda")
        size, taken, refused = 4 * MB, [], 0
        while not refused:                       # tables until nothing is left, the directories' room included
            try:
                taken.append(ctx.table(capacity=size // 4 - 64))
            except wk.WukongError as e:
                assert e.code == wk.E_OOM
                refused += 1
        got = len(taken) * size
        left = torch.cuda.mem_get_info()[0]
        for t in taken:
            t.free()
        del held
        torch.cuda.empty_cache()
        assert got + left > 64 * MB + 4 * MB     # more than was free
        _check(ctx, heavy, qs, o)
        ctx.build_store(tr)
        _check(ctx, heavy, qs, o)


def test_directories_that_a_callers_graph_reads_stay(built):
    import torch
    tr, v = wk.synth_generate(20, seed=0)
    o = oracle.OracleStore(tr)
    q = workloads.heavy_triangle(v)
    want = o.run(q.flat(), q.nvars)[1]
    with wk.Context(0) as ctx:
        ctx.build_store(tr)
        ctx.execute(q)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(torch.cuda.ExternalStream(ctx.stream())):
            graph.capture_begin(capture_error_mode="thread_local")
            ctx.enqueue(q, wk.MODE_RESIDENT)
            graph.capture_end()
            held = torch.empty(torch.cuda.mem_get_info()[0] - 16 * MB, dtype=torch.uint8, device="cuda")
            with pytest.raises(wk.WukongError) as e:
                ctx.table(capacity=17 * MB // 4)
            assert e.value.code == wk.E_OOM
            del held
            torch.cuda.empty_cache()
            graph.replay()
        ctx.check()
        assert _same(ctx.execute(q)[0], want)
        del graph
