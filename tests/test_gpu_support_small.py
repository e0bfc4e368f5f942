"""Support batches from host memory on both sides of the size (2^18 bytes of
candidates) up to which they travel in one pinned copy: results, empty sets, ids
that never occur, refused pointers, and calls of both kinds in turn."""
import numpy as np
import pytest

import oracle
from sgfim import datagen

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def data():
    rows = datagen.regime_txns(5_000, 21, 6, 8, 0.3, seed=2)
    rp, it = datagen.txns_to_csr(rows)
    bm, _ = oracle.build_bitmaps(rp, it, 126)
    return rp, it, bm


# three items a candidate: 20 bytes each, 13,106 candidates are the last small call
@pytest.mark.parametrize("n", [1, 2, 31, 1000, 13_106, 13_107, 13_108, 40_000])
def test_both_sides_of_the_line(engine, data, n):
    rp, it, bm = data
    engine.load_csr(rp, it)
    rng = np.random.default_rng(n)
    items = rng.integers(0, 126, 3 * n).astype(np.uint32)
    ptr = np.arange(n + 1, dtype=np.uint64) * np.uint64(3)
    want = oracle.support_batch(bm, ptr, items)
    assert np.array_equal(engine.support_batch(ptr, items), want)
    small = engine.support_batch(ptr[:3 if n > 1 else 2], items)   # a small call after it
    assert np.array_equal(small, want[:2 if n > 1 else 1])
    assert np.array_equal(engine.support_batch(ptr, items), want)


def test_small_call_odd_candidates(engine, data):
    from sgfim.engine import SgfimError
    rp, it, bm = data
    engine.load_csr(rp, it)
    ptr = np.array([0, 0, 1, 3, 3], np.uint64)
    items = np.array([5, 7, 100_000], np.uint32)   # the empty set, {5}, an id that never occurs, the empty set
    got = engine.support_batch(ptr, items)
    assert list(got) == [5_000, int(oracle.support_batch(bm, np.array([0, 1], np.uint64), items[:1])[0]), 0, 5_000]
    with pytest.raises(SgfimError):
        engine.support_batch(np.array([0, 2, 1, 3], np.uint64), items)
    with pytest.raises(SgfimError):
        engine.support_batch(np.array([1, 2, 3], np.uint64), items)
    assert engine.support_batch(ptr, items)[0] == 5_000
