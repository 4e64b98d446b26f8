"""Row counts the host keeps, result heads that come with the control block, and serving buffers kept
between runs: every writer of a table must be seen, whatever wrote it last."""
import time

import numpy as np
import pytest

import oracle
import workloads
import wukong_b200 as wk

pytestmark = pytest.mark.gpu


def _same(got, want):
    return np.array_equal(oracle.sorted_rows(got), oracle.sorted_rows(want))


def test_row_counts_follow_every_writer(ctx, graph20):
    v, o, inst = graph20["vocab"], graph20["oracle"], graph20["instances"]
    a = np.asarray(inst[v["t_person_a"]], np.uint32).reshape(-1, 1)
    t, out = ctx.table(a), ctx.table()
    for rows in (len(a), 7, 0, 100):
        t.upload(a[:rows])
        assert t.shape() == (rows, 1)
        ctx.known_to_unknown(t, 0, v["p_takes"], wk.OUT, out)
        want = o.step(0, a[:rows], 0, v["p_takes"], wk.OUT)
        assert out.shape() == (len(want), 2) and _same(out.download(), want)
        if rows:
            kept = out.final_process([1], distinct=True)
            final = oracle.final_process(want, [1], distinct=True)   # (merges neighbours of the row order)
            assert kept.shape() == final.shape and np.array_equal(kept.download(), final)
            b = out.filter_bound([0])
            assert b.shape() == out.shape()
            kept.free(), b.free()
    big = ctx.table(capacity=4 * len(want) + 1024)
    ctx.known_to_unknown(t, 0, v["p_takes"], wk.OUT, big)
    t.upload(a[:3])
    assert wk.lib().wk_step_known_to_unknown_noalloc(ctx.h, t.h, 0, v["p_takes"], wk.OUT, big.h) == 0
    assert big.shape()[0] == len(o.step(0, a[:3], 0, v["p_takes"], wk.OUT))
    for x in (t, out, big):
        x.free()


@pytest.mark.parametrize("mode", [wk.MODE_PLAIN, wk.MODE_RESIDENT, wk.MODE_GRAPH])
def test_queries_in_turn(ctx, graph20, mode):
    """Tables below, at and past the head that comes with the control block, the same buffers
    between them, and an enqueued replay whose rows are read afterwards."""
    v, o = graph20["vocab"], graph20["oracle"]
    units = graph20["instances"][v["t_unit"]]
    qs = [workloads.small_chain(v, int(units[0])), workloads.heavy_star(v), workloads.small_chain(v, int(units[5])),
          wk.Query([(v["t_org"], wk.TYPE_ID, wk.IN, -1)]), workloads.heavy_triangle(v),
          wk.Query([(v["t_doc"], wk.TYPE_ID, wk.IN, -1)])]
    buf = np.zeros(1 << 22, np.uint32)
    for q in qs + qs[::-1]:
        _, want, _ = o.run(q.flat(), q.nvars)
        buf[:] = 0xEEEEEEEE
        rows, cols = ctx.execute_host(q, buf, mode)
        assert (rows, cols) == want.shape and _same(buf[:rows * cols].reshape(rows, cols), want)
        got, _ = ctx.execute(q, mode)
        assert _same(got, want)
        if mode != wk.MODE_PLAIN:
            ctx.enqueue(q, mode)
            got, _ = ctx.execute(qs[0], mode)
            assert _same(got, o.run(qs[0].flat(), qs[0].nvars)[1])


def test_serving_runs_in_turn(ctx, graph20):
    """Runs of other sizes, widths and arena sizes on one context, with heavy queries last."""
    v, o = graph20["vocab"], graph20["oracle"]
    for n, seed, arena, heavy in ((40, 1, 0, 2), (200, 2, 0, 0), (10, 3, 1 << 22, 1), (60, 4, 3 << 30, 1), (30, 5, 0, 1)):
        qs = workloads.light_queries(v, graph20["instances"], n, seed=seed, max_len=2 + seed % 5)
        qs += [workloads.heavy_triangle(v)] * heavy
        t0 = time.perf_counter()
        got = ctx.serve(qs, np.zeros(len(qs)), arena_bytes=arena)
        took = time.perf_counter() - t0
        for q, r in zip(qs, got):
            assert r[1] == 0 and _same(r[0], o.run(q.flat(), q.nvars)[1])
    assert took < 0.9   # the last run allocates nothing and ends with its last query
