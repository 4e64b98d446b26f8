"""Index starts of stores whose index keys do not lie where the builder puts them: what a plan takes
from the list is what the start's own step finds, a key behind an empty slot or in a bucket that is not
its own among them, and a key met twice, of which the first on the way counts.  The same for constant
starts."""
import numpy as np
import pytest

import wukong_b200 as wk

pytestmark = pytest.mark.gpu

F = 1 << 17


@pytest.fixture(scope="module")
def graph(built):
    x = np.arange(3000, dtype=np.int64) + F
    tr = np.concatenate([np.stack([x, np.full(3000, 1), 2 + x % 5], 1),
                         np.stack([x, np.full(3000, 10), (x - F + 1) % 3000 + F], 1)]).astype(np.uint32)
    return wk.GStore(tr)


@pytest.mark.parametrize("how", ["whole", "behind_empty", "elsewhere", "twice"])
def test_starts_answer_as_the_probe(graph, how):
    slots, edges, segs = graph.arrays()
    slots = slots.copy()
    index = [s for s in segs if s.index and s.dir == wk.IN][0]
    lo, hi = index.bucket_start * 8, (index.bucket_start + index.num_buckets) * 8
    tids = [t for t in range(2, 7)]
    at = {t: lo + int(np.flatnonzero(slots[lo:hi, 0] == np.uint64(t << 1))[0]) for t in tids}
    if how == "behind_empty":                 # every type's key one slot on, an empty one before it
        for t in tids[:3]:
            b = at[t] // 8 * 8
            slots[b + 1:b + 7] = slots[b:b + 6].copy()
            slots[b] = 0
    elif how == "elsewhere":                  # in the first bucket with room that is not its own
        for t in tids[1:3]:
            row = slots[at[t]].copy()
            b = at[t] // 8 * 8
            keep = [slots[k].copy() for k in range(b, b + 7) if k != at[t]] + [np.zeros(2, np.uint64)]
            slots[b:b + 7] = keep
            other = next(k for k in range(lo, hi, 8) if k != b and slots[k + 6, 0] == 0)
            free = other + int(np.flatnonzero(slots[other:other + 7, 0] == 0)[0])
            slots[free] = row
    elif how == "twice":                      # the same key again in front, with another list
        t = tids[0]
        b = at[t] // 8 * 8
        slots[b + 1:b + 7] = slots[b:b + 6].copy()
        slots[b, 0], slots[b, 1] = t << 1, 3 | (5 << 28)
    with wk.Context(0) as ctx:
        ctx.upload_store(segs, slots, edges)
        seen = 0
        for t in tids:
            first, out = ctx.table(), ctx.table()
            ctx.index_to_unknown(t, wk.IN, first)
            rows = first.download()
            if first.shape()[0]:
                ctx.known_to_unknown(first, 0, 10, wk.OUT, out)
                want = out.download()
            else:
                want = np.zeros((0, 2), np.uint32)
            q = wk.Query([(t, 1, wk.IN, -1), (-1, 10, wk.OUT, -2)])
            for mode in (wk.MODE_PLAIN, wk.MODE_RESIDENT, wk.MODE_GRAPH):
                got = ctx.execute(q, mode)[0]
                assert got.shape == want.shape and np.array_equal(got, want)
            seen += len(rows)
            first.free(), out.free()
        assert seen > 0


@pytest.mark.parametrize("how", ["whole", "behind_empty", "twice"])
def test_constant_starts(graph, how):
    slots, edges, segs = graph.arrays()
    slots = slots.copy()
    starts = [F + 10 * k for k in range(6)]
    for v in starts[:4] if how != "whole" else []:
        at = int(np.flatnonzero(slots[:, 0] == np.uint64(v << 18 | 10 << 1 | wk.OUT))[0])
        b = at // 8 * 8
        if slots[b + 6, 0]:
            continue                          # a full bucket: the key that would fall out matters
        slots[b + 1:b + 7] = slots[b:b + 6].copy()
        slots[b] = 0
        if how == "twice":
            slots[b, 0], slots[b, 1] = v << 18 | 10 << 1 | wk.OUT, 3 | (5 << 28)
    with wk.Context(0) as ctx:
        ctx.upload_store(segs, slots, edges)
        for v in starts:
            first, out = ctx.table(), ctx.table()
            ctx.const_to_unknown(v, 10, wk.OUT, first)
            rows = first.download()
            assert len(rows) == (3 if how == "twice" and v in starts[:4] else 1)
            ctx.known_to_const(first, 0, int(rows[0, 0]) % 5 + 2, 1, wk.OUT, out)
            assert out.shape()[0] >= (how != "twice")
            q = wk.Query([(v, 10, wk.OUT, -1), (-1, 1, wk.OUT, int(rows[0, 0]) % 5 + 2)])
            for mode in (wk.MODE_PLAIN, wk.MODE_RESIDENT, wk.MODE_GRAPH):
                assert np.array_equal(ctx.execute(q, mode)[0], out.download())
            first.free(), out.free()
