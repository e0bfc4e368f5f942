"""Window tasks at the edges of the counting: windows around whole words and
around 32, 64 and 128 words (a lane, two, four words each, and the loop above),
more transactions than 16 bits count, tails of one item up to all 128, items in
every transaction and in none."""
import numpy as np
import pytest

import oracle
from sgfim import datagen

pytestmark = pytest.mark.gpu


def _expect(rows, thr, d):
    rp, it = datagen.txns_to_csr(rows)
    bm, _ = oracle.build_bitmaps(rp, it, d)
    res, _ = oracle.mine_fast(bm, len(rows), thr)
    return {frozenset(s): c for s, c in res}


def _rows(n, d, p, rng):
    """n transactions: item i with probability p[i]."""
    hit = rng.random((n, d)) < np.asarray(p)[None, :]
    return [np.flatnonzero(r).astype(np.uint32) for r in hit]


def _check(rows, d, cap, windows):
    from sgfim.engine import Engine
    from sgfim.service import Ring
    rp, it = datagen.txns_to_csr(rows)
    ring, engine = Ring(d, cap), Engine()
    try:
        ring.append(rp, it)
        res = ring.mine_windows(engine, [s for s, _, _ in windows], [n for _, n, _ in windows],
                                [t for _, _, t in windows])
        assert (res.status == 0).all() and res.batched.all()
        for w, (s, n, thr) in enumerate(windows):
            assert res.as_dict(w) == _expect(rows[s:s + n], thr, d), (w, s, n, thr)
    finally:
        ring.close()
        engine.close()


@pytest.mark.parametrize("d", [1, 2, 5, 31, 64, 65, 127, 128])
def test_window_word_edges(d):
    rng = np.random.default_rng(d)
    p = np.concatenate([[1.0], rng.uniform(0.02, 0.6, d)])[:d]
    if d > 4:
        p[3] = 0.0
        p[4] = 0.97
    rows = _rows(4200, d, p, rng)
    windows = []
    for n in (1, 31, 32, 33, 63, 64, 65, 1023, 1024, 1025, 2047, 2048, 2049, 4095, 4096, 4097):
        s = int(rng.integers(0, len(rows) - n + 1))
        windows.append((s, n, max(1, int(0.3 * n))))
    _check(rows, d, 4200, windows)


@pytest.mark.parametrize("n", [65_534, 65_536, 70_000, 131_072])
def test_window_counts_above_16_bits(n):
    rng = np.random.default_rng(n)
    d = 24
    p = np.concatenate([[1.0, 0.999, 0.99], rng.uniform(0.05, 0.9, d - 3)])
    rows = _rows(n, d, p, rng)
    _check(rows, d, 1 << 17, [(0, n, int(0.25 * n)), (0, n, int(0.6 * n)), (0, n, n), (0, n, int(0.995 * n))])
