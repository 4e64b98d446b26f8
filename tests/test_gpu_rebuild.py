"""A store built again in the same context: its arrays may be the old store's, kept for it, and its
scratch is cut from slabs that are used again within a build.  Every build of a row of sizes up and
down is the one a new context makes, byte for byte, and answers from the new store only."""
import numpy as np
import pytest

import wukong_b200 as wk

pytestmark = pytest.mark.gpu


def _layout(ctx, tr, versatile):
    ctx.build_store(tr, versatile=versatile)
    return ctx.export_store()


@pytest.mark.parametrize("sizes,versatile", [([3, 3, 2, 3, 12, 4, 1, 0, 2], False), ([2, 3, 1, 3], True)])
def test_rebuilt_store_is_a_new_ones(sizes, versatile):
    with wk.Context(0) as kept:
        for seed, orgs in enumerate(sizes):
            tr = wk.synth_generate(orgs, seed=seed)[0] if orgs else np.zeros((0, 3), np.uint32)
            with wk.Context(0) as fresh:
                want = _layout(fresh, tr, versatile)
            got = _layout(kept, tr, versatile)
            assert got[2] == want[2]
            for a, b in zip(got[:2], want[:2]):
                assert a.shape == b.shape and np.array_equal(a, b)


def test_refused_build_then_another():
    tr, _ = wk.synth_generate(3, seed=1)
    with wk.Context(0) as ctx:
        first = _layout(ctx, tr, False)
        with pytest.raises(wk.WukongError):
            ctx.build_store(tr, load_factor=2.0)
        for _ in range(2):
            again = _layout(ctx, tr, False)
            assert again[2] == first[2] and all(np.array_equal(a, b) for a, b in zip(again[:2], first[:2]))
