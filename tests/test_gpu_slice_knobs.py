"""The slice thresholds (knobs 2 and 3) at every length where the way a list is written changes: each
list below, at and above the threshold, in a fused pass and in a fused batch level, row for row against
the oracle; and the defaults read back are the ones in force."""
import numpy as np
import pytest

import oracle
import wukong_b200 as wk

pytestmark = pytest.mark.gpu

F = 1 << 17
OUT, IN = wk.OUT, wk.IN
LENGTHS = (1, 7, 8, 9, 15, 16, 17, 63, 64, 65, 127, 128, 129, 255, 256, 257, 2047, 2048, 2049, 4097)


@pytest.fixture(scope="module")
def lists(built):
    n = 5000
    x = np.arange(n, dtype=np.int64) + F
    tr = [np.stack([x, np.full(n, 1), np.where(x - F < 40 * len(LENGTHS), 2, 3)], 1),
          np.stack([x, np.full(n, 10), (x - F + 1) % n + F], 1)]
    for h, m in enumerate(LENGTHS):               # the hubs lie 40 ids apart, one or two in a warp's rows
        tr.append(np.stack([np.full(m, F + 40 * h), np.full(m, 21), np.arange(m) + F], 1))
    tr = np.concatenate(tr).astype(np.uint32)
    o = oracle.OracleStore(tr)
    with wk.Context(0) as ctx:
        ctx.upload_gstore(wk.GStore(tr))
        yield ctx, o


def test_defaults(built):
    with wk.Context(0) as ctx:
        assert ctx.tune_get(wk.KNOB_SLICE_ROWS) == ctx.tune_get(wk.KNOB_BATCH_SLICE_ROWS) == 128


@pytest.mark.parametrize("thr", [None, 8, 15, 16, 17, 64, 128, 255, 256, 2048, 1 << 23])
def test_lengths_around_the_threshold(lists, thr):
    ctx, o = lists
    q = wk.Query([(2, 1, IN, -1), (-1, 10, OUT, -2), (-1, 21, OUT, -3)])
    want = o.run(q.flat(), q.nvars)[1]
    qs = [wk.Query([(F + 40 * h, 21, OUT, -1), (-1, 10, OUT, -2), (-1, 21, OUT, -3)]) for h in range(len(LENGTHS))]
    if thr:
        ctx.tune_set(wk.KNOB_SLICE_ROWS, thr), ctx.tune_set(wk.KNOB_BATCH_SLICE_ROWS, thr)
    try:
        for mode in (wk.MODE_RESIDENT, wk.MODE_GRAPH):
            assert np.array_equal(ctx.execute(q, mode)[0], want)
        for b, (t, st) in zip(qs, ctx.batch(qs)):
            assert st == 0 and np.array_equal(t, o.run(b.flat(), b.nvars)[1])
    finally:
        ctx.tune_set(wk.KNOB_SLICE_ROWS, 128), ctx.tune_set(wk.KNOB_BATCH_SLICE_ROWS, 128)
