"""Bounded waits that run out within a batch or a serving run: with the spin limit at two polls (knob 6) a
launch gives up waiting and leaves rows unwritten, whose owner queries the next level must not read.  The
call reports the timeout, and with the default limit back the same context answers correctly."""
import numpy as np
import pytest

import oracle
import workloads
import wukong_b200 as wk

pytestmark = pytest.mark.gpu


def _codes(call):
    try:
        call()
        return wk.SUCCESS
    except wk.WukongError as e:
        return e.code


@pytest.mark.parametrize("levels", ["fused", "a pattern each", "flat after tiles"])
def test_levels_after_a_wait_that_ran_out(built, levels):
    tr, v = wk.synth_generate(30, seed=2)
    g = wk.GStore(tr)
    o = oracle.OracleStore(tr)
    inst = {t: g.get_index(t, wk.IN) for t in range(v["t_org"], v["t_doc"] + 1)}
    qs = workloads.light_queries(v, inst, 3000, seed=11)
    want = {k: oracle.sorted_rows(o.run(qs[k].flat(), qs[k].nvars)[1]) for k in range(0, len(qs) - 1, 37)}
    with wk.Context(0) as ctx:
        ctx.upload_gstore(g)
        ctx.tune_set(wk.KNOB_BATCH_FLAT, {"fused": 0, "a pattern each": 1 << 15, "flat after tiles": 0b111100}[levels])
        seen = set()
        for turn in range(6):
            ctx.tune_set(wk.KNOB_SPIN_LIMIT, 2)
            seen.add(_codes(lambda: ctx.batch(qs)))
            seen.add(_codes(lambda: ctx.batch(qs, stream_batch=1000)))
            seen.add(_codes(lambda: ctx.serve(qs, np.zeros(len(qs)))))
            ctx.tune_set(wk.KNOB_SPIN_LIMIT, 0)
            for got in (ctx.batch(qs[:-1]), ctx.batch(qs[:-1], stream_batch=998)) if turn % 3 == 2 else ():
                for k, w in want.items():
                    assert got[k][1] == 0 and np.array_equal(oracle.sorted_rows(got[k][0]), w)
        assert wk.E_TIMEOUT in seen and seen <= {wk.SUCCESS, wk.E_TIMEOUT}, seen
        got = ctx.serve(qs, np.zeros(len(qs)))
        for k, w in want.items():
            assert got[k][1] == 0 and np.array_equal(oracle.sorted_rows(got[k][0]), w)


def test_the_limit_holds_for_a_batch_that_ran_before(built):
    """The captured launches of a batch follow knob 6: the same batch with the limit at two polls and with
    the default again."""
    tr, v = wk.synth_generate(30, seed=2)
    g = wk.GStore(tr)
    inst = {t: g.get_index(t, wk.IN) for t in range(v["t_org"], v["t_doc"] + 1)}
    qs = workloads.light_queries(v, inst, 3000, seed=11)
    with wk.Context(0) as ctx:
        ctx.upload_gstore(g)
        ctx.batch_device(qs)
        codes = []
        for _ in range(4):
            ctx.tune_set(wk.KNOB_SPIN_LIMIT, 2)
            codes.append(_codes(lambda: ctx.batch_device(qs)))
            ctx.tune_set(wk.KNOB_SPIN_LIMIT, 0)
            ctx.batch_device(qs)
        assert wk.E_TIMEOUT in codes
