"""The streamed and the pair-grouped support kernels against the oracle: item counts on both sides of a
record (0, 1, 2, 4, 5, 16, 17, 40), repeated and unknown ids, pairs of one to many candidates (every group
size), row counts on both sides of a staged box, word counts on both sides of a chunk and a step, dense and
sparse rows.  Counts are whole numbers: exact equality."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _bitmaps(n_txn, d, dens, seed):
    rng = np.random.default_rng(seed)
    p = np.exp(rng.uniform(np.log(dens[0]), np.log(dens[1]), d))
    words = (n_txn + 63) // 64
    bits = np.zeros((d, words * 64), bool)
    bits[:, :n_txn] = rng.random((d, n_txn)) < p[:, None]
    return np.ascontiguousarray(np.packbits(bits, axis=1, bitorder="little")).view(np.uint64)


def _candidates(n, d, seed, clustered):
    rng = np.random.default_rng(seed)
    sets = [[], [0], [d - 1], [0, 0], [1, 0, 1], [d + 5], [0, d], list(range(min(d, 16))), list(range(min(d, 17))),
            list(range(min(d, 40)))]
    while len(sets) < n:
        k = int(rng.choice([1, 2, 3, 4, 5, 6, 8, 9, 12, 16, 17]))
        if clustered and rng.random() < 0.8:      # many candidates of few pairs: full groups and every rest
            a = int(rng.integers(0, 3))
            sets.append([a, a + 1] + rng.integers(0, d, max(0, k - 2)).tolist())
        else:
            sets.append(rng.integers(0, d, k).tolist())
    ptr = np.zeros(len(sets) + 1, np.uint64)
    np.cumsum([len(s) for s in sets], out=ptr[1:])
    return ptr, np.array([x for s in sets for x in s], np.uint32)


@pytest.mark.parametrize("kernel", ["pair", "stream", "auto"])
@pytest.mark.parametrize("n_txn,d,n,dens,clustered", [
    (1, 3, 40, (0.5, 1.0), True), (64, 2, 20, (0.1, 0.9), True), (1023, 40, 300, (0.02, 0.2), True),
    (1025, 255, 2000, (0.02, 0.2), False), (16_384, 257, 3000, (0.02, 0.2), True),
    (17_000, 64, 5000, (0.3, 0.9), True), (70_001, 1024, 20_000, (0.02, 0.2), False),
    (33_000, 1792, 4000, (0.01, 0.1), False), (5000, 1793, 500, (0.01, 0.1), False)])
def test_supports_match_oracle(engine, kernel, n_txn, d, n, dens, clustered):
    bm = _bitmaps(n_txn, d, dens, n)
    cp, ci = _candidates(n, d, n + 1, clustered)
    engine.load_bitmaps(bm, n_txn)
    engine.set_support_plan(kernel)
    try:
        got = engine.support_batch(cp, ci)
        again = engine.support_batch(cp[:7], ci)      # a smaller call on the same scratch
    finally:
        engine.set_support_plan("auto")
    known = ci < d
    want = oracle.support_batch(bm, cp, np.where(known, ci, 0).astype(np.uint32))
    for c in range(len(cp) - 1):
        a, b = int(cp[c]), int(cp[c + 1])
        if a == b:
            want[c] = n_txn
        elif not known[a:b].all():
            want[c] = 0
    assert np.array_equal(got, want)
    assert np.array_equal(again, want[:6])


@pytest.mark.parametrize("dens", [(0.02, 0.2), (0.3, 0.9)])
def test_large_auto_calls(engine, dens):
    """A call large enough for the density gate, on both sides of it."""
    n_txn, d, n = 262_144, 300, 500_000
    bm = _bitmaps(n_txn, d, dens, 3)
    rng = np.random.default_rng(4)
    k = rng.integers(1, 12, n)
    cp = np.zeros(n + 1, np.uint64)
    np.cumsum(k, out=cp[1:])
    ci = rng.integers(0, d, int(cp[-1])).astype(np.uint32)
    engine.load_bitmaps(bm, n_txn)
    got = engine.support_batch(cp, ci)
    pick = np.sort(rng.choice(n, 30_000, replace=False))
    sp = np.zeros(len(pick) + 1, np.uint64)
    np.cumsum(k[pick], out=sp[1:])
    si = np.concatenate([ci[int(cp[i]):int(cp[i + 1])] for i in pick])
    assert np.array_equal(got[pick], oracle.support_batch(bm, sp, si))
    engine.set_support_plan("stream")
    try:
        assert np.array_equal(got, engine.support_batch(cp, ci))
    finally:
        engine.set_support_plan("auto")
