"""Fused batch levels (wk_level.cu): batches whose queries run different numbers of steps per level,
against the oracle and the per-pattern levels, with lists on both sides of the slice threshold, runs
longer than a level holds, failing and empty plans, and levels of one row up to several chunks."""
import numpy as np
import pytest

import oracle
import workloads
import wukong_b200 as wk

pytestmark = pytest.mark.gpu

F = 1 << 17


@pytest.fixture(scope="module")
def hub(built):
    """Functional predicates 10..14, and lists by predicate 21 of 1 to 700 entries."""
    n = 3000
    x = np.arange(n, dtype=np.int64) + F
    tr = [np.stack([x, np.full(n, 1), np.full(n, 2)], 1)]
    for k, p in enumerate(range(10, 15)):
        keep = x % (9 + k) != 0
        tr.append(np.stack([x[keep], np.full(keep.sum(), p), (x[keep] - F + 7 * k) % n + F], 1))
    for h, m in enumerate((1, 2, 16, 17, 31, 32, 33, 63, 64, 65, 128, 129, 500, 700)):
        tr.append(np.stack([np.full(m, F + h), np.full(m, 21), np.arange(m) * 2 + F], 1))
    tr = np.concatenate(tr).astype(np.uint32)
    o = oracle.OracleStore(tr)
    with wk.Context(0) as ctx:
        ctx.upload_gstore(wk.GStore(tr))
        yield ctx, o


OUT = wk.OUT


def _queries(n, seed):
    rng = np.random.default_rng(seed)
    qs = []
    for _ in range(n):
        h = int(rng.integers(0, 15))                     # 14: no such list
        steps = [(F + h, 21, OUT, -1)]
        var = 1
        for _ in range(int(rng.integers(0, 7))):
            kind = rng.integers(0, 4)
            s = -int(rng.integers(1, var + 1))
            if kind == 0 and var < 7:
                steps.append((s, 10 + int(rng.integers(0, 5)), OUT, -(var + 1)))
                var += 1
            elif kind == 1 and var < 7 and rng.random() < 0.4:
                steps.append((s, 21, OUT, -(var + 1)))
                var += 1
            elif kind == 2:
                steps.append((s, 1, OUT, 2))
            elif var > 1:
                steps.append((s, 10 + int(rng.integers(0, 5)), OUT, -int(rng.integers(1, var + 1))))
        qs.append(wk.Query(steps, nvars=8))
    return qs


@pytest.mark.parametrize("n,seed", [(1, 1), (2, 2), (33, 3), (700, 4)])
@pytest.mark.parametrize("thr", [8, 64, 1 << 20])
def test_mixed_runs(hub, n, seed, thr):
    ctx, o = hub
    qs = _queries(n, seed)
    qs[n // 2:n // 2] = [wk.Query([]), wk.Query([(-1, 10, OUT, -2)])]   # nothing to do; starts unbound
    ctx.tune_set(wk.KNOB_BATCH_SLICE_ROWS, thr)
    try:
        fused = ctx.batch(qs)
        ctx.tune_set(wk.KNOB_BATCH_FLAT, 1 << 15)                       # a pattern per level
        plain = ctx.batch(qs)
    finally:
        ctx.tune_set(wk.KNOB_BATCH_FLAT, 0)
        ctx.tune_set(wk.KNOB_BATCH_SLICE_ROWS, 128)
    for q, (a, sa), (b, sb) in zip(qs, fused, plain):
        st, want, _ = o.run(q.flat(), q.nvars)
        assert sa == sb == st
        if st == 0 and q.patterns:
            assert np.array_equal(a, want) and np.array_equal(b, want)


def test_many_rows(hub):
    """Levels of several chunks per CTA, as one batch and as a stream of batches."""
    ctx, o = hub
    qs = [wk.Query([(F + 13, 21, OUT, -1), (-1, 10, OUT, -2), (-2, 21, OUT, -3), (-3, 1, OUT, 2)], nvars=3)] * 300
    qs += [wk.Query([(F + 12, 21, OUT, -1), (-1, 21, OUT, -2), (-2, 11, OUT, -3)], nvars=3)] * 900
    want = {id(q): o.run(q.flat(), q.nvars)[1] for q in (qs[0], qs[-1])}
    for got in (ctx.batch(qs), ctx.batch(qs, stream_batch=500)):
        for q, (t, st) in zip(qs, got):
            assert st == 0 and np.array_equal(t, want[id(q)])
