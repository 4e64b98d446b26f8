"""Serving buffers kept between runs: made once, given back with the store, to an allocation that needs
them, and at the end of a run on a device that has little room besides."""
import numpy as np
import pytest

import oracle
import workloads
import wukong_b200 as wk

pytestmark = pytest.mark.gpu

GB = 1 << 30


@pytest.fixture(scope="module")
def small(built):
    tr, v = wk.synth_generate(3, seed=8)
    g = wk.GStore(tr)
    inst = {t: g.get_index(t, wk.IN) for t in range(v["t_org"], v["t_doc"] + 1)}
    qs = workloads.light_queries(v, inst, 40, seed=1) + [workloads.heavy_triangle(v)]
    o = oracle.OracleStore(tr)
    want = [oracle.sorted_rows(o.run(q.flat(), q.nvars)[1]) for q in qs]
    return g, tr, qs, want


def _serve(ctx, qs, want):
    for r, w in zip(ctx.serve(qs, np.zeros(len(qs))), want):
        assert r[1] == 0 and np.array_equal(oracle.sorted_rows(r[0]), w)


def _free():
    import torch
    return torch.cuda.mem_get_info()[0]


def test_a_later_run_allocates_nothing(small):
    g, _, qs, want = small
    with wk.Context(0) as ctx:
        ctx.upload_gstore(g)
        _serve(ctx, qs, want)
        _serve(ctx, qs, want)
        before = wk.device_allocs()
        _serve(ctx, qs, want)
        assert wk.device_allocs() == before


@pytest.mark.parametrize("load", ["upload", "build"])
def test_given_back_with_the_store(small, load):
    g, tr, qs, want = small
    with wk.Context(0) as ctx:
        ctx.upload_gstore(g)
        before = _free()
        _serve(ctx, qs, want)
        assert before - _free() > 2 * GB       # the arenas
        ctx.upload_gstore(g) if load == "upload" else ctx.build_store(tr)
        assert before - _free() < GB // 2
        _serve(ctx, qs, want)


def test_given_back_on_a_full_device(small):
    import torch
    g, _, qs, want = small
    with wk.Context(0) as ctx:
        ctx.upload_gstore(g)
        _serve(ctx, qs, want)
        held = torch.empty(_free() - 1 * GB, dtype=torch.uint8, device="cuda")
        t = ctx.table(capacity=(2 * GB) // 4)  # fits only in the arenas' place
        t.free()
        del held
        torch.cuda.empty_cache()
        held = torch.empty(_free() - 12 * GB, dtype=torch.uint8, device="cuda")
        before = _free()
        _serve(ctx, qs, want)
        assert before - _free() < GB // 2      # an eighth of 12 GB would not hold them
        del held
        torch.cuda.empty_cache()
        assert ctx.measure_random_reads(1 << 20, 1) > 0
