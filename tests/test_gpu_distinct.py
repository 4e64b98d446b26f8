"""DISTINCT by keys alone (the columns up to the last required one fit 64 bits) beside the general
sort (they do not, or more than 32 columns are required), against the oracle: widths at the edge
of a key, tile and CTA remainders, columns that no longer take part, constant columns, values past
2^31, and a window of the result."""
import numpy as np
import pytest

import oracle
import wukong_b200 as wk

pytestmark = pytest.mark.gpu


def _table(n, bits, seed):
    """One column per entry: that many bits between its smallest and its largest value."""
    rng = np.random.default_rng(seed)
    cols = []
    for b in bits:
        base = 0 if b == 32 else int(rng.integers(0, 2**31 - 2**b)) + 2**31 * int(rng.integers(0, 2))
        c = (base + rng.integers(0, 2**b, n)).astype(np.uint32)
        lo, hi = (2**31, 2**31 - 1) if b == 32 else (base, base + 2**b - 1)   # (signed order)
        c[rng.integers(0, n)] = lo
        if n > 1 and b:
            c[np.flatnonzero(c != lo)[:1]] = hi
        cols.append(c)
    t = np.stack(cols, axis=1)
    return np.concatenate([t, t[rng.integers(0, n, n // 3)]])[rng.permutation(n + n // 3)]


@pytest.mark.parametrize("bits,keep", [
    ([32, 32], [0, 1]),                # a full key
    ([32, 32, 1], [0, 1, 2]),          # one bit past it: the general sort
    ([32, 32, 32], [1]),               # the last column orders nothing that is output
    ([32, 32, 7], [2, 0]),
    ([3, 0, 9, 20], [2, 1, 2]),        # a constant column, a column twice
    ([0, 0, 5], [1]),                  # only constant columns matter: the table is in order
    ([1], [0]),
    ([8, 8], [1]),                     # neighbours are merged, not all equal values
    ([4, 4, 4], [0, 1] * 17),          # 34 required columns: the general sort
])
@pytest.mark.parametrize("n", [2, 1535, 1536, 1537, 40000])   # with the repeats: 2,046 to 2,049 rows
def test_distinct_matches_the_oracle(bits, keep, n):
    t = _table(n, bits, seed=n + len(keep))
    with wk.Context(0) as ctx:
        tin = ctx.table(t)
        for offset, limit in ((0, -1), (3, 700), (n // 5, -1), (2 * n, 5)):
            got = tin.final_process(keep, distinct=True, offset=offset, limit=limit).download()
            want = oracle.final_process(t, keep, distinct=True, offset=offset, limit=limit)
            assert got.shape == want.shape and np.array_equal(got, want), (offset, limit)


@pytest.mark.parametrize("extra", [0, 1])
def test_distinct_with_more_than_one_tile_a_cta(extra):
    """148 x 8 tiles of 2,048 rows, and one row more."""
    n = 148 * 8 * 2048 + extra
    rng = np.random.default_rng(extra)
    t = np.stack([rng.integers(0, 300, n), rng.integers(2**31 - 2000, 2**31 + 2000, n)], axis=1).astype(np.uint32)
    with wk.Context(0) as ctx:
        got = ctx.table(t).final_process([0, 1], distinct=True).download()
    assert np.array_equal(got, oracle.final_process(t, [0, 1], distinct=True))
