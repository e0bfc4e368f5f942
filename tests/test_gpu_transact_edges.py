"""Quantile selection and window medians at the edges of their kernels: every median network and its
neighbours, columns that are constant, tied, signed zero or infinite, more ranks than one select batch
or histogram group holds, more sensors than a transpose tile, row counts around the tiles.  Exact
equality with the numpy restatement."""
import numpy as np
import pytest

from oracle import online, transact

pytestmark = pytest.mark.gpu


def _vals(n, S, seed):
    rng = np.random.default_rng(seed)
    v = np.round(np.cumsum(rng.integers(-20, 21, (n, S)), axis=0) + rng.integers(-300, 301, (n, S))) / 1000.0
    if S > 1:
        v[:, 1] = rng.integers(-1, 2, n) * 0.0           # signed zeros
        v[::3, 1] = -1e-300
    if S > 2:
        v[:, 2] = 4.0
    if S > 3:
        v[:, 3] = rng.standard_normal(n) * 1e200
        v[:: max(1, n // 7), 3] = np.inf
        v[1:: max(1, n // 5), 3] = -np.inf
    return v


@pytest.mark.parametrize("window", [1, 2, 15, 16, 17, 31, 32, 33, 63, 64, 65, 256])
def test_window_medians(engine, window):
    vals = _vals(3000, 3, window)
    items, labels, edges = engine.transactionize(vals, window, max(1, window // 3), 5)
    want_edges = transact.fit_bins(vals, 5)
    assert all(np.array_equal(a, b) for a, b in zip(edges, want_edges))
    want, _ = transact.window_items(vals, want_edges, window, max(1, window // 3), None, 5)
    assert np.array_equal(items, want)
    if window <= 64:
        o_items, _, o_edges = engine.transactionize_online(vals[:600], window, window, 4)
        w_edges, w_items, _ = online.online_items(vals[:600], window, window, 4, None)
        assert np.array_equal(o_items, w_items)
        assert np.array_equal(o_edges.view(np.int64), w_edges.view(np.int64))


@pytest.mark.parametrize("n,S,bins", [(1, 1, 3), (2, 3, 2), (63, 2, 6), (64, 33, 3), (65, 31, 4), (8191, 4, 7),
                                      (8193, 4, 1), (20_000, 5, 700), (30_001, 70, 16)])
def test_quantile_edges(engine, n, S, bins):
    vals = _vals(n, S, n + bins)
    with np.errstate(all="ignore"):
        q = np.quantile(vals, np.linspace(0, 1, bins + 1), axis=0)
    if np.isnan(q).any():      # between two infinities numpy's interpolation is NaN: keep those columns finite
        vals[:, 3] = np.clip(vals[:, 3], -1e200, 1e200)
    _, _, edges = engine.transactionize(vals, 1, max(1, n // 50), bins)
    want = transact.fit_bins(vals, bins)
    for a, b in zip(edges, want):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n", [65_535, 65_536, 200_001])
def test_quantiles_with_and_without_lists(engine, n):
    """Columns long enough that the later passes read a list of the values left (spread values), and
    columns that crowd under the open prefixes so that no list holds them: constant, a few values,
    values that differ in the last bits only, half constant and half spread."""
    rng = np.random.default_rng(n)
    v = np.empty((n, 6))
    v[:, 0] = rng.standard_normal(n)
    v[:, 1] = 3.25
    v[:, 2] = rng.integers(0, 5, n) / 7.0
    v[:, 3] = 1.0 + rng.integers(0, 1 << 20, n) * 2.0 ** -52
    v[:, 4] = np.where(rng.random(n) < 0.5, -2.0, rng.random(n) * 1e6)
    v[:, 5] = rng.random(n) * 10.0 ** rng.integers(-200, 200, n)
    _, _, edges = engine.transactionize(v, 1, n // 50, 6)
    for a, b in zip(edges, transact.fit_bins(v, 6)):
        assert np.array_equal(a, b)
    _, _, edges = engine.transactionize(v, 1, n // 50, 40)   # more ranks than a histogram group
    for a, b in zip(edges, transact.fit_bins(v, 40)):
        assert np.array_equal(a, b)
