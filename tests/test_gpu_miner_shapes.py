"""The wave miner's kernels at the edges of their tiles: transactions around whole
words, 256-word chunks and segments; items sparse enough for listed projections
(at most 10 bits a word), dense enough for compressed ones, and both in one
dataset; against the oracle, with and without projections, and with an arena too
small for every node's mask."""
import numpy as np
import pytest

import oracle
from sgfim import datagen

pytestmark = pytest.mark.gpu

DENSITY = {"sparse": (0.02, 0.15), "dense": (0.3, 0.9), "mixed": (0.02, 0.95)}


def _rows(n, d, kind, rng):
    lo, hi = DENSITY[kind]
    p = np.exp(rng.uniform(np.log(lo), np.log(hi), d))
    p[0] = 1.0
    group = rng.random((n, 1)) < 0.5   # items that come together, so that sets grow
    hit = rng.random((n, d)) < np.where(group, np.minimum(1.0, 1.6 * p), 0.4 * p)[:, :]
    hit[:, 0] = True
    return [np.flatnonzero(r).astype(np.uint32) for r in hit]


@pytest.mark.parametrize("kind,d,frac", [("sparse", 40, 0.01), ("dense", 12, 0.1), ("mixed", 18, 0.05)])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 127, 129, 16_383, 16_384, 16_385, 70_001])
def test_miner_edges_match_oracle(n, kind, d, frac):
    from sgfim.engine import Engine
    rng = np.random.default_rng(n + d)
    rows = _rows(n, d, kind, rng)
    thr = max(1 if n < 65 else 3, int(np.ceil(frac * n)))
    rp, it = datagen.txns_to_csr(rows)
    bm, _ = oracle.build_bitmaps(rp, it, d)
    want = {frozenset(s): c for s, c in oracle.mine_fast(bm, n, thr)[0]}
    for projection in (True, False):
        for wave in (0, 7):
            with Engine(projection=projection, wave_nodes=wave) as eng:
                got = eng.load_csr(rp, it).mine(thr)
                assert got.as_dict() == want, (projection, wave)


@pytest.mark.parametrize("projection", [True, False])
def test_miner_small_arena_matches_oracle(projection):
    """64 mask slots (the least): most nodes run without a mask."""
    from sgfim.engine import Engine
    n, d = 300_000, 24
    rng = np.random.default_rng(5)
    rows = _rows(n, d, "mixed", rng)
    rp, it = datagen.txns_to_csr(rows)
    bm, _ = oracle.build_bitmaps(rp, it, d)
    thr = int(0.04 * n)
    want = {frozenset(s): c for s, c in oracle.mine_fast(bm, n, thr)[0]}
    with Engine(projection=projection, hbm_budget=8 << 20) as eng:
        assert eng.load_csr(rp, it).mine(thr).as_dict() == want
