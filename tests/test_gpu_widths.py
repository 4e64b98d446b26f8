"""Passes and batch levels that multiply rows of wide tables, up to the 32 columns a table may have:
lists on both sides of what a lane, the warp's stage and the slice queue take (16, 17, 256, 257
entries), alone in a warp and mixed, as single steps over tables of 65,536 rows and more and as whole
queries, row for row against the oracle."""
import numpy as np
import pytest

import oracle
import wukong_b200 as wk

pytestmark = pytest.mark.gpu

F = 1 << 17
OUT, IN = wk.OUT, wk.IN
LENGTHS = (1, 16, 17, 256, 257)


@pytest.fixture(scope="module")
def wide(built):
    """n vertices of one type, functional predicates 10..12, and lists by predicate 21 of LENGTHS
    entries, the first of which are the vertices with lists themselves."""
    n = 600
    x = np.arange(n, dtype=np.int64) + F
    tr = [np.stack([x, np.full(n, 1), np.full(n, 2)], 1)]
    for k, p in enumerate((10, 11, 12)):
        tr.append(np.stack([x, np.full(n, p), (x - F + 11 * k + 1) % n + F], 1))
    for h, m in enumerate(LENGTHS):
        tr.append(np.stack([np.full(m, F + h), np.full(m, 21), np.arange(m) + F], 1))
    tr = np.concatenate(tr).astype(np.uint32)
    o = oracle.OracleStore(tr)
    with wk.Context(0) as ctx:
        ctx.upload_gstore(wk.GStore(tr))
        yield ctx, o, n


@pytest.mark.parametrize("w_out", [8, 16, 17, 24, 32])
@pytest.mark.parametrize("rows", [65536, 65541])
def test_single_steps(wide, w_out, rows):
    ctx, o, n = wide
    rng = np.random.default_rng(w_out)
    t = rng.integers(F + len(LENGTHS), F + n, size=(rows, w_out - 1), dtype=np.int64).astype(np.uint32)
    cs = w_out // 2
    for h in range(len(LENGTHS)):                       # 512 rows where the warps meet one length each,
        t[1024 * h:1024 * h + 512:37, cs] = F + h       # one row of it or two at a time
    t[8192:8704:5, cs] = F + rng.integers(0, len(LENGTHS), 103)
    t[-3:, cs] = F + 2
    tin, out = ctx.table(t), ctx.table()
    ctx.known_to_unknown(tin, cs, 21, OUT, out)
    got, want = out.download(), o.step(0, t, cs, 21, OUT)
    tin.free(), out.free()
    assert got.shape[1] == w_out and np.array_equal(got, want)


def _wide_query(first, w_out):
    """From `first`, functional steps up to w_out - 1 columns, then the lists of the first one."""
    steps = [first] + [(-1, 10 + j % 3, OUT, -2 - j) for j in range(w_out - 2)] + [(-1, 21, OUT, -w_out)]
    return wk.Query(steps, nvars=w_out)


@pytest.mark.parametrize("w_out", [8, 16, 17, 24, 32])
def test_whole_queries(wide, w_out):
    ctx, o, _ = wide
    for first in ((2, 1, IN, -1), (F + 4, 21, OUT, -1), (F + 2, 21, OUT, -1)):
        q = _wide_query(first, w_out)
        st, want, _ = o.run(q.flat(), q.nvars)
        assert st == 0 and want.shape[1] == w_out and len(want)
        for mode in (wk.MODE_PLAIN, wk.MODE_RESIDENT, wk.MODE_GRAPH):
            assert np.array_equal(ctx.execute(q, mode)[0], want)


@pytest.mark.parametrize("w_out", [8, 15, 16])
def test_batch_levels(wide, w_out):
    """A batch takes 16 patterns a query, so 16 columns."""
    ctx, o, _ = wide
    qs = [_wide_query((F + h, 21, OUT, -1), w_out) for h in (4, 0, 3, 1, 2)] * 3
    for got in (ctx.batch(qs), ctx.batch(qs, stream_batch=4)):
        for q, (t, st) in zip(qs, got):
            assert st == 0 and np.array_equal(t, o.run(q.flat(), q.nvars)[1])
