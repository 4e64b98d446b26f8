"""Plans whose rows hold vertex 0, which names a predicate's index list, in a step on a functional
predicate: a store whose lists hold the id 0 (as an uploaded one may) in a one-entry list, a short, a
long and a chunked one.  Every way to run, time or enqueue such a plan takes the index list's rows, on
the first call already.  And a predicate that has two segments, whose lists are in only one of them."""
import numpy as np
import pytest

import oracle
import wukong_b200 as wk

pytestmark = pytest.mark.gpu

F = 1 << 17
OUT, IN = wk.OUT, wk.IN
N = 12000
LISTS = {"one": (10, 1), "short": (20, 6), "long": (21, 40), "chunk": (22, 9000)}


def _graph():
    x = np.arange(N, dtype=np.int64) + F
    tr = [np.stack([x, np.full(N, 1), np.full(N, 2)], 1)]
    for k, p in enumerate((10, 11, 12)):
        m = N if p == 10 else 300
        tr.append(np.stack([x[:m], np.full(m, p), (x[:m] - F + 7 * k + 1) % N + F], 1))
    for p, m in ((20, 6), (21, 40), (22, 9000)):
        tr.append(np.stack([np.full(m, F + 5), np.full(m, p), np.arange(m) + F], 1))
        tr.append(np.stack([x[7:90], np.full(83, p), x[7:90]], 1))
    return np.concatenate(tr).astype(np.uint32)


@pytest.fixture(scope="module", params=list(LISTS))
def zeroed(request, built):
    tr = _graph()
    o = oracle.OracleStore(tr)
    pid, length = LISTS[request.param]
    g = wk.GStore(tr)
    slots, edges, segs = g.arrays()
    edges = edges.copy()
    key = (F + 5) << 18 | pid << 1 | OUT
    ptr = int(slots[np.flatnonzero(slots[:, 0] == key)[0], 1])
    at, size = (ptr >> 28) & ((1 << 34) - 1), ptr & ((1 << 28) - 1)
    assert size == length
    edges[at] = 0
    q = wk.Query([(F + 5, 11, OUT, -1), (-1, 11, IN, -2), (-2, pid, OUT, -3), (-3, 11, OUT, -4), (-3, 12, OUT, -5)])
    t = o.run([x for x in wk.Query(q.patterns[:2]).flat()], 2)[1]
    t = o.step(0, t, 1, pid, OUT)
    t[0, 2] = 0
    for p in (11, 12):
        t = o.step(0, t, 2, p, OUT)
    assert len(t) >= 300 * 300                  # the index lists of 11 and 12 for the row of vertex 0
    yield (segs, slots, edges), q, t            # (views of g, which lives as long)
    g.close()


MODES = [wk.MODE_PLAIN, wk.MODE_RESIDENT, wk.MODE_GRAPH]


@pytest.mark.parametrize("flat_rows", [1, 65536, 0])
def test_queries(zeroed, flat_rows):
    store, q, want = zeroed
    with wk.Context(0) as ctx:
        ctx.upload_store(*store)
        ctx.tune_set(wk.KNOB_FLAT_ROWS, flat_rows)
        prof = ctx.profile(q, iters=1)
        assert prof[-1]["rows_out"] == len(want)
        for mode in MODES:
            assert np.array_equal(ctx.execute(q, mode)[0], want)
            if mode != wk.MODE_PLAIN:
                ctx.enqueue(q, mode)
                ctx.check()


def test_enqueue_first(zeroed):
    """Enqueued on buffers that another plan has sized, before the plan itself has run."""
    store, q, want = zeroed
    with wk.Context(0) as ctx:
        ctx.upload_store(*store)
        sizing = wk.Query([(2, 1, IN, -1), (-1, 10, OUT, -2), (-1, 1, OUT, 2)])
        ctx.execute(sizing)
        ctx.enqueue(q, wk.MODE_RESIDENT)
        ctx.check()


def test_batches_and_serving(zeroed):
    store, q, want = zeroed
    start = wk.Query([(2, 1, IN, -1), (-1, 1, OUT, 2)])
    with wk.Context(0) as ctx:
        ctx.upload_store(*store)
        qs = [q, wk.Query([(F + 9, 10, OUT, -1), (-1, 10, OUT, -2)]), q]
        for got in (ctx.batch(qs), ctx.batch(qs, stream_batch=2)):
            for k in (0, 2):
                assert got[k][1] == 0 and np.array_equal(got[k][0], want)
        for r in (ctx.serve([q, start, q], np.zeros(3)),):
            for k in (0, 2):
                assert r[k][1] == 0 and np.array_equal(oracle.sorted_rows(r[k][0]), oracle.sorted_rows(want))


def test_a_predicate_in_two_segments(built):
    tr = _graph()
    o = oracle.OracleStore(tr)
    g = wk.GStore(tr)
    slots, edges, segs = g.arrays()
    segs = list(segs)
    segs += [s for s in segs if not s.index and s.pid in (20, 21, 22)]
    arr = (wk.SegMeta * len(segs))(*segs)
    q = wk.Query([(2, 1, IN, -1), (-1, 20, OUT, -2), (-2, 21, OUT, -3), (-3, 10, OUT, -4)])
    want = o.run(q.flat(), q.nvars)[1]
    with wk.Context(0) as ctx:
        ctx.upload_store(arr, slots, edges)
        assert ctx.profile(q, iters=1)[-1]["rows_out"] == len(want)
        for mode in MODES:
            assert np.array_equal(ctx.execute(q, mode)[0], want)
        t, st = ctx.batch([q])[0]
        assert st == 0 and np.array_equal(t, want)
