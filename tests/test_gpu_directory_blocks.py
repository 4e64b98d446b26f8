"""Lookups at the edges of a directory's blocks (32 ids each) and of its range, row for row in the
reference's order: ids on both sides of every multiple of 32, with a key or without, in segments whose
range begins and ends inside a block, at every step and launch that reads a directory."""
import numpy as np
import pytest

import oracle
import wukong_b200 as wk

pytestmark = pytest.mark.gpu

F = 1 << 17
OUT = wk.OUT


@pytest.fixture(scope="module", params=[0, 1, 31, 45])
def store(request, built):
    n, first = 2000, F + request.param
    x = np.arange(n, dtype=np.int64) + first
    keep = {10: (x % 32 != 31), 20: (x % 64 != 32) & (x % 96 != 63), 21: (x % 32 == 0) | (x % 32 == 31)}
    tr = [np.stack([x, np.full(n, 1), np.full(n, 2)], 1),
          np.stack([x[keep[10]], np.full(keep[10].sum(), 10), (x[keep[10]] - first + 33) % n + first], 1)]
    for p in (20, 21):
        for j in range(3):
            s = x[keep[p]]
            tr.append(np.stack([s, np.full(len(s), p), (s - first) % 89 + first + 100 * j], 1))
    tr = np.concatenate(tr).astype(np.uint32)
    o = oracle.OracleStore(tr)
    with wk.Context(0) as ctx:
        ctx.upload_gstore(wk.GStore(tr))
        yield ctx, o, first, n


@pytest.mark.parametrize("flat_rows", [0, 1])
@pytest.mark.parametrize("lanes", [1, 4])
def test_steps_in_order(store, flat_rows, lanes):
    ctx, o, first, n = store
    edges = np.arange(first // 32 * 32, first + n + 96, 32)
    v = np.concatenate([edges - 1, edges, edges + 1, [first - 1, first, first + n - 1, first + n, F - 5, 0xFFFFFFFF]])
    t = np.stack([np.arange(len(v)), v, np.roll(v, 7)], 1).astype(np.uint32)
    ctx.tune_set(wk.KNOB_LANES, lanes), ctx.tune_set(wk.KNOB_FLAT_ROWS, flat_rows)
    try:
        tin, out = ctx.table(t), ctx.table()
        for pid in (10, 20, 21, 1):
            ctx.known_to_unknown(tin, 1, pid, OUT, out)
            assert np.array_equal(out.download(), o.step(0, t, 1, pid, OUT))
            ctx.known_to_known(tin, 1, 2, pid, OUT, out)
            assert np.array_equal(out.download(), o.step(1, t, 1, pid, OUT, ce=2))
            ctx.known_to_const(tin, 1, first + 133, pid, OUT, out)
            assert np.array_equal(out.download(), o.step(2, t, 1, pid, OUT, end_const=first + 133))
        tin.free(), out.free()
    finally:
        ctx.tune_set(wk.KNOB_LANES, 2), ctx.tune_set(wk.KNOB_FLAT_ROWS, 65536)


def test_plans_and_batches_in_order(store):
    ctx, o, first, n = store
    qs = [wk.Query([(int(s), 20, OUT, -1), (-1, 10, OUT, -2), (-2, 21, OUT, -3), (-3, 1, OUT, 2)])
          for s in range(max(F, first // 32 * 32 - 1), first + 200)]
    qs.append(wk.Query([(2, 1, wk.IN, -1), (-1, 10, OUT, -2), (-2, 21, OUT, -3), (-3, 10, OUT, -4)]))
    for q, (t, st) in zip(qs, ctx.batch(qs)):
        want = o.run(q.flat(), q.nvars)[1]
        assert st == 0 and np.array_equal(t, want)
    for q in qs[::9] + qs[-1:]:
        for mode in (wk.MODE_RESIDENT, wk.MODE_GRAPH):
            assert np.array_equal(ctx.execute(q, mode)[0], o.run(q.flat(), q.nvars)[1])
