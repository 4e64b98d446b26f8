"""A predicate whose keys all have empty lists, as an uploaded store may hold them, in the segment whose
directory words come last: its directory has blocks but no words, and a lookup that finds no key must
have a word to load all the same."""
import numpy as np
import pytest

import oracle
import wukong_b200 as wk

pytestmark = pytest.mark.gpu

F = 1 << 17


@pytest.mark.parametrize("all_empty", [True, False])
def test_lookups_in_a_segment_without_words(built, all_empty):
    n = 4000
    x = np.arange(n, dtype=np.int64) + F
    tr = [np.stack([x, np.full(n, 1), np.full(n, 2)], 1)]
    for k, p in enumerate((10, 11, 12)):
        tr.append(np.stack([x, np.full(n, p), (x - F + 7 * k + 1) % n + F], 1))
    tr = np.concatenate(tr).astype(np.uint32)
    g = wk.GStore(tr)
    slots, edges, segs = g.arrays()
    slots = slots.copy()
    last = max((s for s in segs if not s.index and s.num_buckets), key=lambda s: s.bucket_start)
    key = slots[:, 0]
    data = (np.arange(len(key)) % 8 != 7) & (key & np.uint64((1 << 18) - 1) == last.pid * 2 + last.dir)
    if not all_empty:
        data &= (key >> np.uint64(18)) % np.uint64(3) == 0
    slots[data, 1] &= ~np.uint64((1 << 28) - 1)             # the lists' lengths
    emptied = set((key[data] >> np.uint64(18)).tolist())
    d = int(last.dir)
    of = {int(r[0 if d else 2]): int(r[2 if d else 0]) for r in tr[tr[:, 1] == last.pid]}
    tab = np.stack([np.arange(n + 40, dtype=np.uint32), np.arange(n + 40, dtype=np.uint32) + F - 20], 1)
    want = np.array([[a, v, of[v]] for a, v in tab.tolist() if v in of and v not in emptied], np.uint32).reshape(-1, 3)
    with wk.Context(0) as ctx:
        ctx.upload_store(segs, slots, edges)
        for flat_rows in (1, 65536):
            ctx.tune_set(wk.KNOB_FLAT_ROWS, flat_rows)
            tin, out = ctx.table(tab), ctx.table()
            ctx.known_to_unknown(tin, 1, last.pid, d, out)
            assert np.array_equal(out.download(), want)
            ctx.known_to_const(tin, 1, F + 5, last.pid, d, out)
            assert np.array_equal(out.download(), want[want[:, 2] == F + 5][:, :2])
            tin.free(), out.free()
