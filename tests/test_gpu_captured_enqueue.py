"""A plan enqueued while the caller captures the context's stream: each replay of that graph writes the
context's tables without the host, so their row counts are read anew whatever was read in between."""
import ctypes as C

import numpy as np
import pytest

import oracle
import workloads
import wukong_b200 as wk

pytestmark = pytest.mark.gpu


def test_row_counts_follow_a_callers_replays(built):
    import torch
    tr, v = wk.synth_generate(3, seed=6)
    o = oracle.OracleStore(tr)
    g = wk.GStore(tr)
    units = g.get_index(v["t_unit"], wk.IN)
    plans = [workloads.small_chain(v, int(u)) for u in units[:2]]
    want = [o.run(q.flat(), q.nvars)[1] for q in plans]
    assert len(want[0]) != len(want[1])
    with wk.Context(0) as ctx:
        ctx.upload_gstore(g)
        table, rows = C.c_void_p(), C.c_uint64()

        def run(k):
            qc = plans[k].as_c()
            assert wk.lib().wk_query_execute(ctx.h, C.byref(qc), wk.MODE_RESIDENT, C.byref(table), None, None,
                                             C.byref(rows)) == 0
            return rows.value

        def shape():
            r, c = C.c_uint64(), C.c_int32()
            assert wk.lib().wk_table_shape(ctx.h, table, C.byref(r), C.byref(c)) == 0
            return r.value, c.value

        run(0), run(1)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(torch.cuda.ExternalStream(ctx.stream())):
            graph.capture_begin(capture_error_mode="thread_local")
            ctx.enqueue(plans[0], wk.MODE_RESIDENT)
            graph.capture_end()
            for _ in range(3):
                assert run(1) == len(want[1]) and shape() == want[1].shape
                graph.replay()
                assert shape() == want[0].shape
                got = np.zeros(want[0].size, np.uint32)
                assert wk.lib().wk_table_download(ctx.h, table, got.ctypes.data_as(C.c_void_p), got.size) == 0
                assert np.array_equal(oracle.sorted_rows(got.reshape(want[0].shape)), oracle.sorted_rows(want[0]))
        del graph
