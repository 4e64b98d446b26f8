"""Vertex directories (wk_dir.cu) against the oracle: dense ids (every segment has a directory),
sparse ids (none has: the hash probes at every group width), and a mix, with start ids at the
edges of a directory's range and of its 64-id blocks; stores whose chains or keys are not as the
builder leaves them; and a context whose store is replaced."""
import numpy as np
import pytest

import oracle
import workloads
import wukong_b200 as wk

pytestmark = pytest.mark.gpu

BLANK = 0xFFFFFFFF
FIRST = 1 << 17


def _relabel(tr, f):
    tr = tr.copy()
    tr[:, 0] = f(tr[:, 0])
    o = tr[:, 2]
    tr[:, 2] = np.where(o >= FIRST, f(o), o)
    return tr


def _same(got, want):
    return np.array_equal(oracle.sorted_rows(got), oracle.sorted_rows(want))


KINDS = {
    "dense": lambda x: x + 29,                                       # ranges begin inside a block
    "sparse": lambda x: FIRST + (x - FIRST) * 9001,                  # no segment is worth one
    "mixed": lambda x: np.where(x % 3 == 0, x, FIRST + (x - FIRST) * 300),   # some are
}


@pytest.fixture(scope="module", params=list(KINDS))
def store(request, built):
    tr, v = wk.synth_generate(4, seed=3)
    tr = _relabel(tr.astype(np.int64), KINDS[request.param]).astype(np.uint32)
    o = oracle.OracleStore(tr)
    g = wk.GStore(tr, load_factor=0.3)
    inst = {t: g.get_index(t, wk.IN) for t in range(v["t_org"], v["t_doc"] + 1)}
    with wk.Context(0) as ctx:
        ctx.upload_gstore(g)
        yield {"ctx": ctx, "v": v, "o": o, "tr": tr, "inst": inst}


def _starts(tr, pid):
    s = np.unique(tr[tr[:, 1] == pid, 0]).astype(np.int64)
    edge = np.concatenate([s[:3], s[-3:], s[:1] - 1, s[-1:] + 1, s[-1:] + 64, (s // 64) * 64, (s // 64) * 64 + 63,
                           [0, 5, BLANK]])
    v = np.concatenate([s, edge, s[::-1]])
    return v[(v >= 0) & (v <= BLANK)].astype(np.uint32)


@pytest.mark.parametrize("lanes", [1, 2, 4, 8])
@pytest.mark.parametrize("flat_rows", [0, 1])
def test_steps(store, lanes, flat_rows):
    ctx, v, o, tr = store["ctx"], store["v"], store["o"], store["tr"]
    ctx.tune_set(wk.KNOB_LANES, lanes)
    ctx.tune_set(wk.KNOB_FLAT_ROWS, flat_rows)
    try:
        for pid in (v["p_member_of"], v["p_takes"], v["p_sub_org_of"], v["p_author"], wk.TYPE_ID):
            starts = _starts(tr, pid)
            tab = np.stack([np.arange(len(starts), dtype=np.uint32), starts], axis=1)
            objs = tr[tr[:, 1] == pid, 2]
            filt = np.stack([starts, np.resize(objs, len(starts))], axis=1)
            with_in = wk.OUT
            for op in (0, 1, 2):
                t_in = tab if op != 1 else filt
                cs = 1 if op != 1 else 0
                want = o.step(op, t_in, cs, pid, with_in, ce=1, end_const=int(objs[0]))
                tin, out = ctx.table(t_in), ctx.table()
                if op == 0:
                    ctx.known_to_unknown(tin, cs, pid, with_in, out)
                elif op == 1:
                    ctx.known_to_known(tin, cs, 1, pid, with_in, out)
                else:
                    ctx.known_to_const(tin, cs, int(objs[0]), pid, with_in, out)
                got = out.download()
                assert np.array_equal(got, want) or _same(got, want), (pid, op)
                tin.free(), out.free()
    finally:
        ctx.tune_set(wk.KNOB_LANES, 2)
        ctx.tune_set(wk.KNOB_FLAT_ROWS, 65536)


@pytest.mark.parametrize("lanes,flat", [(1, 0), (4, 0), (2, 63)])
def test_batch(store, lanes, flat):
    ctx, v, o = store["ctx"], store["v"], store["o"]
    qs = workloads.light_queries(v, store["inst"], 150, seed=4)
    ctx.tune_set(wk.KNOB_BATCH_LANES, lanes)
    ctx.tune_set(wk.KNOB_BATCH_FLAT, flat)
    try:
        for q, (t, st) in zip(qs, ctx.batch(qs)):
            _, want, _ = o.run(q.flat(), q.nvars)
            assert st == 0 and _same(t, want)
    finally:
        ctx.tune_set(wk.KNOB_BATCH_LANES, 4)
        ctx.tune_set(wk.KNOB_BATCH_FLAT, 0)


def _chained(built_tr):
    g = wk.GStore(built_tr, load_factor=1.0)
    slots, edges, segs = g.arrays()
    return g, slots.copy(), edges.copy(), segs


@pytest.mark.parametrize("fault", ["link", "twice"])
def test_malformed_stores_answer_as_the_probe(built, fault):
    """A chain link past the slot array is reported when a probe follows it; of a key stored
    twice in a bucket the first counts."""
    tr, v = wk.synth_generate(2, seed=5)
    o = oracle.OracleStore(tr)
    g, slots, edges, segs = _chained(tr) if fault == "link" else (None, None, None, None)
    if fault == "twice":
        g = wk.GStore(tr)
        slots, edges, segs = g.arrays()
        slots = slots.copy()
        k = slots[:, 0].reshape(-1, 8)
        one = np.flatnonzero((k[:, 0] != 0) & (k[:, 1] == 0))[::3]
        slots[one * 8 + 1, 0] = slots[one * 8, 0]
        slots[one * 8 + 1, 1] = 1 | (7 << 28)   # another list: edge 7 alone
    else:
        k = slots[:, 0].reshape(-1, 8)
        linked = np.flatnonzero(k[:, 7] != 0)
        slots[linked * 8 + 7, 0] = np.uint64(len(k) + 5) << np.uint64(18)
    persons = np.concatenate([g.get_index(v[t], wk.IN) for t in ("t_person_a", "t_person_b", "t_person_c")])
    persons = np.ascontiguousarray(persons.reshape(-1, 1))
    with wk.Context(0) as ctx:
        ctx.upload_store(segs, slots, edges)
        tin, out = ctx.table(persons), ctx.table()
        if fault == "link":
            with pytest.raises(wk.WukongError) as e:
                ctx.known_to_unknown(tin, 0, v["p_takes"], wk.OUT, out)
            assert e.value.code == wk.E_CORRUPT
        else:
            ctx.known_to_unknown(tin, 0, v["p_takes"], wk.OUT, out)
            assert _same(out.download(), o.step(0, persons, 0, v["p_takes"], wk.OUT))
        tin.free(), out.free()


def test_replaced_store(built):
    """Another store in the same context: queries, captured graphs, batches and serving lanes
    answer from the new one."""
    with wk.Context(0) as ctx:
        for n, seed in ((2, 1), (3, 2), (2, 1)):
            tr, v = wk.synth_generate(n, seed=seed)
            o = oracle.OracleStore(tr)
            ctx.build_store(tr)
            heavy = workloads.heavy_star(v)
            g = wk.GStore(tr)
            inst = {t: g.get_index(t, wk.IN) for t in range(v["t_org"], v["t_doc"] + 1)}
            qs = workloads.light_queries(v, inst, 60, seed=9)
            for mode in (wk.MODE_RESIDENT, wk.MODE_GRAPH):
                _, want, _ = o.run(heavy.flat(), heavy.nvars)
                assert _same(ctx.execute(heavy, mode)[0], want)
            mixed = qs[:30] + [heavy] + qs[30:]
            for q, (t, st) in zip(qs, ctx.batch(qs)):
                assert st == 0 and _same(t, o.run(q.flat(), q.nvars)[1])
            for q, r in zip(mixed, ctx.serve(mixed, np.zeros(len(mixed)))):
                assert r[1] == 0 and _same(r[0], o.run(q.flat(), q.nvars)[1])
