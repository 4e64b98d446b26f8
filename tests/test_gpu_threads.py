"""Contexts in several threads: one captures its batches and plans while others load stores and grow
their buffers.  A wait for the whole device in one thread would end another's capture."""
import threading
import time

import numpy as np
import pytest

import oracle
import workloads
import wukong_b200 as wk

pytestmark = pytest.mark.gpu


def test_captures_loads_and_growing_buffers_at_once(built):
    tr, v = wk.synth_generate(6, seed=1)
    g = wk.GStore(tr)
    o = oracle.OracleStore(tr)
    inst = {t: g.get_index(t, wk.IN) for t in range(v["t_org"], v["t_doc"] + 1)}
    qs = workloads.light_queries(v, inst, 240, seed=3)
    heavy = [workloads.heavy_star(v), workloads.heavy_triangle(v)]
    want = [oracle.sorted_rows(o.run(q.flat(), q.nvars)[1]) for q in qs]
    hwant = [oracle.sorted_rows(o.run(q.flat(), q.nvars)[1]) for q in heavy]
    end, bad = time.perf_counter() + 6, []

    def work(seed):
        rng = np.random.default_rng(seed)
        try:
            while time.perf_counter() < end and not bad:
                with wk.Context(0, rbuf_bytes=1 << 16) as ctx:      # (everything grows again)
                    for _ in range(4):
                        ctx.build_store(tr) if rng.random() < 0.5 else ctx.upload_gstore(g)
                        n = int(rng.integers(1, len(qs)))
                        for got in (ctx.batch(qs[:n]), ctx.batch(qs[:n], stream_batch=max(1, n // 3))):
                            for (t, st), w in zip(got, want):
                                assert st == 0 and np.array_equal(oracle.sorted_rows(t), w)
                        for q, w in zip(heavy, hwant):
                            assert np.array_equal(oracle.sorted_rows(ctx.execute(q, wk.MODE_GRAPH)[0]), w)
                        for r, w in zip(ctx.serve(qs[:20] + heavy[:1], np.zeros(21), arena_bytes=1 << 22),
                                        want[:20] + hwant[:1]):
                            assert r[1] == 0 and np.array_equal(oracle.sorted_rows(r[0]), w)
        except Exception as e:
            bad.append((seed, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(5)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
