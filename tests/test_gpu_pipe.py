"""Fused passes of a single query (wk_pipe.cu) against the oracle, row for row: runs of functional
steps and filters longer than a pass holds, one and several rounds per chunk, lists on both sides of
the row-by-row and the slice thresholds, a start list of one entry, and rows of vertex 0."""
import numpy as np
import pytest

import oracle
import wukong_b200 as wk

pytestmark = pytest.mark.gpu

F = 1 << 17


@pytest.fixture(scope="module")
def chain(built):
    """n vertices, functional predicates 10..15 (x -> x + n * k), predicate 20 with lists of 0 to 3
    entries, and hubs whose lists by predicate 21 have 200, 257 and 5000 entries."""
    n = 40000
    x = np.arange(n, dtype=np.int64) + F
    tr = [np.stack([x, np.full(n, 1), np.full(n, 2)], 1)]
    for k, p in enumerate(range(10, 16)):
        keep = x % (7 + k) != 0                      # some vertices have no value
        tr.append(np.stack([x[keep], np.full(keep.sum(), p), x[keep] + n * (k + 1)], 1))
    for j in range(3):
        keep = x % 4 > j
        tr.append(np.stack([x[keep], np.full(keep.sum(), 20), x[keep] % 997 + F + j], 1))
    for h, m in ((5, 200), (6, 257), (7, 5000), (8, 1)):
        tr.append(np.stack([np.full(m, F + h), np.full(m, 21), np.arange(m) * 3 + F + 11], 1))
    tr.append(np.array([[F + 9, 1, 3]]))             # a type with one instance
    tr = np.concatenate(tr).astype(np.uint32)
    o = oracle.OracleStore(tr)
    with wk.Context(0) as ctx:
        ctx.upload_gstore(wk.GStore(tr))
        yield ctx, o, n


def _check(ctx, o, q):
    st, want, _ = o.run(q.flat(), q.nvars)
    for mode in (wk.MODE_RESIDENT, wk.MODE_GRAPH):
        got, _ = ctx.execute(q, mode)
        assert st == 0 and np.array_equal(got, want)


OUT, IN = wk.OUT, wk.IN
FUNC = [(-1, 10 + k, OUT, -2 - k) for k in range(6)]


@pytest.mark.parametrize("steps", [FUNC[:1], FUNC[:3], FUNC[:4], FUNC,                     # columns past a pass
                                   [(-1, 1, OUT, 2)] * 7,                                  # steps past a pass
                                   FUNC[:2] + [(-1, 20, OUT, -4), (-4, 20, OUT, -5)],      # two expansions
                                   FUNC[:2] + [(-1, 10, OUT, -2), (-1, 11, OUT, -3), (F + 6, 21, OUT, -1)]])
def test_runs_of_steps(chain, steps):
    ctx, o, _ = chain
    _check(ctx, o, wk.Query([(2, 1, IN, -1)] + steps))


@pytest.mark.parametrize("thr", [8, 128, 4000])
def test_list_lengths(chain, thr):
    ctx, o, _ = chain
    ctx.tune_set(wk.KNOB_SLICE_ROWS, thr)
    try:
        for tail in ([], [(-2, 10, OUT, -3)]):
            _check(ctx, o, wk.Query([(21, 0, IN, -1), (-1, 21, OUT, -2)] + tail))
            _check(ctx, o, wk.Query([(2, 1, IN, -1), (-1, 11, OUT, -3), (-1, 21, OUT, -2)] + [(-2, 12, OUT, -4)]))
    finally:
        ctx.tune_set(wk.KNOB_SLICE_ROWS, 128)


def test_one_entry_starts(chain):
    ctx, o, _ = chain
    for first in ((3, 1, IN, -1), (F + 8, 21, OUT, -1)):
        for tail in ([(-1, 20, OUT, -2)], [(-1, 11, OUT, -2)], [(-1, 1, OUT, 2)], [(-1, 21, OUT, -2)]):
            _check(ctx, o, wk.Query([first] + tail))


@pytest.mark.parametrize("rows", [1, 31, 257, 65536, 303104, 303105, 700001])
def test_rows_per_chunk(chain, rows):
    """Single steps over tables of one row up to several rounds per chunk, vertex 0 (which names an
    index), blank and absent ids among them."""
    ctx, o, n = chain
    rng = np.random.default_rng(rows)
    t = rng.integers(F, F + n, size=(rows, 2), dtype=np.int64).astype(np.uint32)
    t[::50, 1] = 0xFFFFFFFF
    t[3::50, 1] = F + 3 * n
    if rows < 1000:
        t[7::29, 1] = 0
    ctx.tune_set(wk.KNOB_FLAT_ROWS, 1)
    try:
        tin, out = ctx.table(t), ctx.table()
        for pid in (10, 20):
            ctx.known_to_unknown(tin, 1, pid, OUT, out)
            assert np.array_equal(out.download(), o.step(0, t, 1, pid, OUT))
        t[:, 0] = np.where(rng.random(rows) < 0.5, t[:, 1] + n, t[:, 0])
        tin.upload(t)
        ctx.known_to_known(tin, 1, 0, 10, OUT, out)
        assert np.array_equal(out.download(), o.step(1, t, 1, 10, OUT, ce=0))
        ctx.known_to_const(tin, 1, F + 5, 20, OUT, out)
        assert np.array_equal(out.download(), o.step(2, t, 1, 20, OUT, end_const=F + 5))
        tin.free(), out.free()
    finally:
        ctx.tune_set(wk.KNOB_FLAT_ROWS, 65536)
