"""Calls that launch without asking for results, on a context whose store is gone: a load that failed
leaves no store, and nothing of the one before it may reach a launch."""
import numpy as np
import pytest

import oracle
import workloads
import wukong_b200 as wk

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def stores(built):
    tr, v = wk.synth_generate(3, seed=4)
    g = wk.GStore(tr)
    slots, edges, segs = g.arrays()
    bad = slots.copy()
    full = np.flatnonzero((bad[:, 0] != 0) & (np.arange(len(bad)) % 8 != 7))
    bad[full[0], 1] = 5 | (np.uint64(len(edges)) << np.uint64(28))   # a list past the edge array
    return {"v": v, "g": g, "o": oracle.OracleStore(tr), "bad": (segs, bad, edges)}


def _lose_store(ctx, stores):
    with pytest.raises(wk.WukongError) as e:
        ctx.upload_store(*stores["bad"])
    assert e.value.code == wk.E_CORRUPT


def test_enqueue(stores):
    q = workloads.heavy_star(stores["v"])
    want = stores["o"].run(q.flat(), q.nvars)[1]
    with wk.Context(0) as ctx:
        ctx.upload_gstore(stores["g"])
        for mode in (wk.MODE_RESIDENT, wk.MODE_GRAPH):
            ctx.execute(q, mode)
        _lose_store(ctx, stores)
        for mode in (wk.MODE_RESIDENT, wk.MODE_GRAPH):
            with pytest.raises(wk.WukongError):
                ctx.enqueue(q, mode)
        assert wk.lib().wk_query_enqueue(ctx.h, q.as_c(), wk.MODE_RESIDENT) == wk.E_NOSTORE
        ctx.check()
        ctx.upload_gstore(stores["g"])
        assert np.array_equal(oracle.sorted_rows(ctx.execute(q)[0]), oracle.sorted_rows(want))


def test_enqueue_before_any_store(stores):
    q = workloads.heavy_star(stores["v"])
    with wk.Context(0) as ctx:
        assert wk.lib().wk_query_enqueue(ctx.h, q.as_c(), wk.MODE_RESIDENT) == wk.E_NOSTORE


def test_batch_replay(stores):
    """The last batch's graph launches on the store and the scratch of its time: not once they are gone."""
    v, o = stores["v"], stores["o"]
    inst = {t: stores["g"].get_index(t, wk.IN) for t in range(v["t_org"], v["t_doc"] + 1)}
    qs = workloads.light_queries(v, inst, 50, seed=2)
    with wk.Context(0) as ctx:
        ctx.upload_gstore(stores["g"])
        ctx.batch_device(qs)
        ctx.batch_replay()
        ctx.check()
        ctx.upload_gstore(stores["g"])
        assert wk.lib().wk_batch_replay(ctx.h) == wk.E_BADARG
        for q, (t, st) in zip(qs, ctx.batch(qs)):
            assert st == 0 and np.array_equal(oracle.sorted_rows(t), oracle.sorted_rows(o.run(q.flat(), q.nvars)[1]))
        ctx.batch_replay()
        ctx.check()
        big = ctx.table(np.full((1 << 22, 1), 1 << 17, np.uint32), capacity=1 << 23)   # more tiles than the scratch has words
        out = ctx.table(capacity=1 << 27)                                              # and more slices
        ctx.known_to_const(big, 0, 1 << 17, v["p_takes"], wk.OUT, out)
        ctx.known_to_unknown(big, 0, v["p_takes"], wk.OUT, out)
        rc = wk.lib().wk_batch_replay(ctx.h)
        assert rc == wk.E_BADARG
        ctx.check()
        big.free(), out.free()
        _lose_store(ctx, stores)
        assert wk.lib().wk_batch_replay(ctx.h) == wk.E_BADARG
