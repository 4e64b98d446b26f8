"""A store whose chains do not end (every linked bucket's chain leads back to itself): it loads, gets no
directories, and a probe that follows such a chain reports it; keys in the buckets themselves are found."""
import numpy as np
import pytest

import wukong_b200 as wk

pytestmark = pytest.mark.gpu


def test_chains_that_do_not_end(built):
    tr, v = wk.synth_generate(2, seed=5)
    g = wk.GStore(tr, load_factor=1.0)
    slots, edges, segs = g.arrays()
    slots = slots.copy()
    key = slots[:, 0].reshape(-1, 8)
    linked = np.flatnonzero(key[:, 7] != 0)
    assert len(linked) > 100
    slots[linked * 8 + 7, 0] = linked.astype(np.uint64) << np.uint64(18)
    persons = np.concatenate([g.get_index(v[t], wk.IN) for t in ("t_person_a", "t_person_b", "t_person_c")])
    with wk.Context(0) as ctx:
        ctx.upload_store(segs, slots, edges)
        tin, out = ctx.table(np.ascontiguousarray(persons.reshape(-1, 1))), ctx.table()
        with pytest.raises(wk.WukongError) as e:
            ctx.known_to_unknown(tin, 0, v["p_takes"], wk.OUT, out)
        assert e.value.code == wk.E_CORRUPT
        k = slots[:, 0].reshape(-1, 8)[:, :7]
        home = k[(k & np.uint64((1 << 18) - 1)) == np.uint64(v["p_takes"] * 2 + wk.OUT)] >> np.uint64(18)
        found = 0
        for p in np.intersect1d(home, persons.astype(np.uint64))[:20]:
            tin.upload(np.array([[p]], np.uint32))
            try:
                ctx.known_to_unknown(tin, 0, v["p_takes"], wk.OUT, out)
            except wk.WukongError as err:            # (moved to a chain's later bucket)
                assert err.code == wk.E_CORRUPT
                continue
            want = tr[(tr[:, 0] == p) & (tr[:, 1] == v["p_takes"]), 2]
            assert np.array_equal(out.download()[:, 1], np.unique(want))
            found += 1
        assert found
        tin.free(), out.free()
