"""The work this engine is used for, as cases that can be timed and compared.

Every case goes through the Python front end (``sgfim.engine``, ``sgfim.service``,
``sgfim.mlp``).  The families and what they stand for:

* ``support``    counting the supports of a batch of candidate itemsets: through
                 host arrays on a loaded dataset, or on device pointers for a
                 caller whose bitmaps already sit in HBM.  Two kinds of data: wide,
                 sparse item spaces with random-walk candidates, and sensor states
                 (one bin per sensor) with candidates that do occur together.
* ``cooc``       the pairwise co-occurrence matrix of the bitmap rows.
* ``mine``       a new transaction set loaded and its maximal frequent itemsets
                 mined: what one call of the engine adapter does.
* ``anytime``    mining of a large dataset that is already resident.
* ``windows``    a batch of sliding windows of the service's ring, mined in one call.
* ``train``      loss and gradients of the extension scorer on a batch of trace rows.
* ``score``      the extension scorer's probabilities for a wave of extensions.
* ``transact``   a sensor stream turned into transactions: quantile bins, or online
                 (P2) edges per window.

``model`` seeds the process that produces the data (regime weights and tables: one
plant, one machine); the preparation's seed draws the stream from it.  Where the
result is a set of itemsets, whose number would change with the draw, the model seeds
the draw too, and the preparation's seed says in which order its transactions (or
windows) come and which sensor state has which item id.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "20261008-self-growing-evidence-agent_gb300"))

from sgfim.engine import Engine  # noqa: E402
from sgfim.mlp import Trainer, to_bf16_bits  # noqa: E402
from sgfim.service import Ring  # noqa: E402

DEV = "cuda"
GB = 1 << 30


def listed():
    return [
        # an analyst's handful of itemsets on the small dataset: the call's latency
        dict(name="support-host-small", kind="support", data="sensors", api="host", n_txn=20_000, sensors=8, bins=5,
             regimes=4, alpha=0.3, n_cand=200, kmin=1, kmax=5, model=0),
        # a search front's candidates on sensor states: dense rows, sets that occur, some longer than eight
        dict(name="support-sensors", kind="support", data="sensors", api="device", n_txn=300_007, sensors=80, bins=8,
             regimes=32, alpha=0.2, n_cand=65_536, kmin=2, kmax=10, model=0),
        # the benchmark's workload: a million random-walk candidates over 1,024 sparse items
        dict(name="support-1m", kind="support", data="sparse", api="device", n_txn=1 << 20, items=1024, regimes=16,
             n_cand=1_000_000, kmin=3, kmax=8, model=0),
        # co-occurrence of one service window (126 items): launch-bound
        dict(name="cooc-window", kind="cooc", data="sensors", n_txn=65_536, sensors=21, bins=6, regimes=8, alpha=0.3,
             model=0),
        # co-occurrence of the benchmark's bitmaps
        dict(name="cooc-1024", kind="cooc", data="sparse", n_txn=1 << 20, items=1024, regimes=16, model=0),
        # the small mining configuration from loading to the result (floor 1%)
        dict(name="mine-small", kind="mine", n_txn=20_000, sensors=8, bins=5, regimes=4, alpha=0.3, floor=0.01,
             order="support", model=0),
        # the large mining configuration at a floor whose set is complete in well under a second
        dict(name="anytime-2m", kind="anytime", n_txn=2_000_000, sensors=80, bins=8, regimes=32, alpha=0.2, floor=0.03,
             model=0),
        # what one scheduler of the window service takes from its queue at 2,000 requests/s
        dict(name="windows-batch", kind="windows", n_win=45, len_lo=512, len_hi=65_536, floor=0.02, model=0),
        # a backlog of windows mined at full load
        dict(name="windows-backlog", kind="windows", n_win=768, len_lo=512, len_hi=65_536, floor=0.02, model=0),
        # one training step's gradients of the extension scorer at the trainer's batch size
        dict(name="train-4096", kind="train", rows=4096, hidden=128),
        # the extensions of a wide search wave scored at once
        dict(name="score-wave", kind="score", rows=300_000, hidden=128),
        # a fleet stream of a million rows discretised at its quantiles
        dict(name="transact-1m", kind="transact", rows=1_000_000, sensors=21, bins=6, window=30, stride=15,
             online=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["support", "support", "cooc", "mine", "anytime", "windows", "train", "score", "transact"])
    model = rng.randrange(1, 1000)
    if kind == "support":
        if rng.random() < 0.5:
            return dict(kind=kind, data="sparse", api="device", n_txn=_log(rng, 1 << 14, 1 << 20),
                        items=_log(rng, 64, 1400), regimes=16, n_cand=_log(rng, 1000, 600_000), kmin=3, kmax=8,
                        model=model)
        return dict(kind=kind, data="sensors", api=rng.choice(["host", "device"]), n_txn=_log(rng, 5_000, 1_000_000),
                    sensors=rng.randrange(8, 81), bins=rng.randrange(4, 9), regimes=rng.randrange(4, 33), alpha=0.3,
                    n_cand=_log(rng, 100, 200_000), kmin=rng.randrange(1, 4), kmax=rng.randrange(5, 11), model=model)
    if kind == "cooc":
        if rng.random() < 0.5:
            return dict(kind=kind, data="sparse", n_txn=_log(rng, 1 << 15, 1 << 20), items=_log(rng, 64, 1400),
                        regimes=16, model=model)
        return dict(kind=kind, data="sensors", n_txn=_log(rng, 5_000, 1_000_000), sensors=rng.randrange(8, 81),
                    bins=rng.randrange(4, 9), regimes=rng.randrange(4, 33), alpha=0.3, model=model)
    if kind == "mine":
        return dict(kind=kind, n_txn=_log(rng, 3_000, 100_000), sensors=rng.randrange(6, 13), bins=rng.randrange(4, 7),
                    regimes=rng.randrange(4, 9), alpha=0.3, floor=round(rng.uniform(0.01, 0.04), 4),
                    order=rng.choice(["support", "support_desc"]), model=model)
    if kind == "anytime":
        return dict(kind=kind, n_txn=_log(rng, 200_000, 1_500_000), sensors=rng.randrange(40, 81),
                    bins=rng.randrange(6, 9), regimes=32, alpha=0.2, floor=round(rng.uniform(0.04, 0.06), 4),
                    model=model)
    if kind == "windows":
        lo = _log(rng, 300, 4096)
        return dict(kind=kind, n_win=_log(rng, 1, 400), len_lo=lo, len_hi=_log(rng, 2 * lo, 50_000),
                    floor=round(rng.uniform(0.02, 0.05), 4), model=rng.randrange(0, 4))
    if kind == "train":
        return dict(kind=kind, rows=_log(rng, 500, 20_000), hidden=rng.choice([64, 128, 128, 256]))
    if kind == "score":
        return dict(kind=kind, rows=_log(rng, 1_000, 250_000), hidden=rng.choice([64, 128, 128]))
    online = rng.random() < 0.4
    window = rng.randrange(10, 61)
    return dict(kind=kind, rows=_log(rng, 20_000, 700_000), sensors=rng.randrange(3, 25), bins=rng.randrange(3, 9),
                window=window, stride=rng.randrange(window // 3, window + 1), online=online)


# ------------------------------------------------------------------ data
def _items_of(case):
    return case["items"] if case.get("data") == "sparse" else case["sensors"] * case["bins"]


def _words(n_txn):
    return ((n_txn + 63) // 64 + 1) & ~1   # the engine's rows are whole 16-byte pieces


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _pack(bits, n_words):
    """bool [rows, n] -> int64 [rows, n_words]: bit t & 63 of word t >> 6 is column t."""
    r, n = bits.shape
    full = torch.zeros((r, n_words * 64), dtype=torch.uint8, device=DEV)
    full[:, :n] = bits
    w = torch.tensor([1, 2, 4, 8, 16, 32, 64, 128], dtype=torch.uint8, device=DEV)
    return (full.view(r, -1, 8) * w).sum(2, dtype=torch.uint8).contiguous().view(torch.int64)


def _sensor_tables(case):
    rng = np.random.default_rng(case["model"])
    w = rng.dirichlet(np.ones(case["regimes"]))
    p = rng.dirichlet(np.full(case["bins"], case["alpha"]), size=(case["regimes"], case["sensors"]))
    cdf = np.cumsum(p, axis=2)
    cdf[:, :, -1] = 1.0
    return torch.tensor(np.cumsum(w), device=DEV, dtype=torch.float32), torch.tensor(cdf, device=DEV, dtype=torch.float32)


def _sensor_bins(case, seed, n):
    """uint8 [n, sensors]: the bin of every sensor in every transaction."""
    cw, cdf = _sensor_tables(case)
    g = _gen(seed)
    z = torch.searchsorted(cw, torch.rand(n, generator=g, device=DEV)).clamp_(max=len(cw) - 1)
    out = torch.empty((n, case["sensors"]), dtype=torch.uint8, device=DEV)
    for s in range(case["sensors"]):
        u = torch.rand(n, generator=g, device=DEV)
        out[:, s] = (u[:, None] >= cdf[z, s, :-1]).sum(1, dtype=torch.uint8)
    return out


def _sensor_bitmaps(bins, case, n_words):
    rows = [_pack(torch.stack([bins[:, s] == b for b in range(case["bins"])]), n_words)
            for s in range(case["sensors"])]
    return torch.cat(rows)


def _shuffled(bins, seed):
    return bins[torch.randperm(len(bins), generator=_gen(seed), device=DEV)]


def _sensor_items(bins, case, seed):
    """uint32 [n, sensors], ascending, on the host: the seed's ids of the states (sensor, bin)."""
    d = case["sensors"] * case["bins"]
    ids = torch.tensor(np.random.default_rng(seed).permutation(d), device=DEV, dtype=torch.int32)
    base = torch.arange(case["sensors"], device=DEV, dtype=torch.int32) * case["bins"]
    out = np.empty((len(bins), case["sensors"]), np.uint32)
    for a in range(0, len(bins), 1 << 18):
        out[a:a + (1 << 18)] = ids[bins[a:a + (1 << 18)].to(torch.int32) + base].sort(1)[0].cpu().numpy()
    return out


def _sparse_bitmaps(case, seed):
    """Marginals log-uniform in [2%, 20%], correlated through the regimes."""
    rng = np.random.default_rng(case["model"])
    w = rng.dirichlet(np.ones(case["regimes"]))
    m = np.exp(rng.uniform(np.log(0.02), np.log(0.20), size=case["items"]))
    a = rng.exponential(1.0, size=(case["regimes"], case["items"]))
    p = np.minimum(1.0, m[None, :] * a / (w @ a)[None, :])
    g = _gen(seed)
    n, n_words = case["n_txn"], _words(case["n_txn"])
    cw = torch.tensor(np.cumsum(w), device=DEV, dtype=torch.float32)
    z = torch.searchsorted(cw, torch.rand(n, generator=g, device=DEV)).clamp_(max=len(cw) - 1)
    pt = torch.tensor(p.T.copy(), device=DEV, dtype=torch.float32)
    step = max(1, (1 << 27) // n)
    return torch.cat([_pack(torch.rand((min(step, case["items"] - e), n), generator=g, device=DEV)
                            < pt[e:e + step][:, z], n_words) for e in range(0, case["items"], step)])


def _csr(sets, k):
    """Padded sets [n, kmax] (ascending, the valid ones first) and sizes k -> CSR."""
    ptr = np.zeros(len(k) + 1, np.uint64)
    np.cumsum(k, out=ptr[1:])
    keep = np.arange(sets.shape[1])[None, :] < k[:, None]
    return ptr, np.ascontiguousarray(sets[keep], dtype=np.uint32)


def _walk_sets(case, rng):
    """Distinct random items, 3 to 8 of them: the random walk of a sparse pair graph."""
    n, d, kmax = case["n_cand"], case["items"], case["kmax"]
    s = rng.integers(0, d, size=(n, kmax))
    while True:
        o = np.sort(s, axis=1)
        bad = np.nonzero((o[:, 1:] == o[:, :-1]).any(axis=1))[0]
        if not len(bad):
            break
        s[bad] = rng.integers(0, d, size=(len(bad), kmax))
    k = rng.integers(case["kmin"], kmax + 1, size=n)
    s[np.arange(kmax)[None, :] >= k[:, None]] = 1 << 30
    return _csr(np.sort(s, axis=1), k)


def _occurring_sets(case, rng, bins):
    """States of random sensors in random transactions: sets that occur."""
    n, kmax = case["n_cand"], min(case["kmax"], case["sensors"])
    t = torch.tensor(rng.integers(0, bins.shape[0], size=n), device=DEV)
    of = bins[t].cpu().numpy()
    sensors = np.argsort(rng.random((n, case["sensors"]), dtype=np.float32), axis=1)[:, :kmax]
    k = rng.integers(min(case["kmin"], kmax), kmax + 1, size=n)
    s = sensors * case["bins"] + np.take_along_axis(of, sensors, axis=1)
    s[np.arange(kmax)[None, :] >= k[:, None]] = 1 << 30
    return _csr(np.sort(s, axis=1), k)


def _stream(case, seed):
    """[rows, sensors] float64 on the host: levels that wander, a cycle and noise, in thousandths (ties occur)."""
    g = _gen(seed)
    n, S = case["rows"], case["sensors"]
    t = torch.arange(n, device=DEV, dtype=torch.float64)[:, None]
    level = torch.cumsum(torch.randint(-20, 21, (n, S), generator=g, device=DEV), 0)
    period = torch.randint(50, 400, (1, S), generator=g, device=DEV).double()
    cycle = ((t % period) - torch.floor(period / 2)).abs() * 8
    noise = torch.randint(-300, 301, (n, S), generator=g, device=DEV)
    vals = torch.round(level + cycle + noise) / 1000.0
    anomaly = (torch.rand(n, generator=g, device=DEV) < 0.05).to(torch.int32)
    return vals.cpu().numpy(), anomaly.cpu().numpy()


def _scorer(case, seed):
    """Trace rows, labels, weights and the network's parameters (weights are bf16 values)."""
    rng = np.random.default_rng(seed)
    n, h = case["rows"], case["hidden"]
    x = rng.random((n, 8), dtype=np.float32)
    x[:, 4] = rng.integers(1, 12, n) / 16.0                       # depth / 16
    x[:, :3] *= 0.2                                               # supports as fractions
    y = (rng.random(n) < 0.74).astype(np.float32)
    wt = np.where(y > 0.5, 0.5 / 0.74, 0.5 / 0.26).astype(np.float32)

    def bf16(a):
        return (to_bf16_bits(a).astype(np.uint32) << 16).view(np.float32)
    p = {"W1": bf16(rng.uniform(-1, 1, (h, 8)) * np.sqrt(3.0 / 8)), "b1": rng.normal(0, 0.05, h).astype(np.float32),
         "W2": bf16(rng.uniform(-1, 1, (h, h)) * np.sqrt(3.0 / h)), "b2": rng.normal(0, 0.05, h).astype(np.float32),
         "w3": bf16(rng.uniform(-1, 1, h) * np.sqrt(3.0 / h)), "b3": rng.normal(0, 0.05, 1).astype(np.float32)}
    return x, y, wt, p


# ------------------------------------------------------------------ cases
def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind in ("support", "cooc"):
        n, n_words = case["n_txn"], _words(case["n_txn"])
        bins = None
        if case["data"] == "sparse":
            bm = _sparse_bitmaps(case, seed)
        else:
            bins = _sensor_bins(case, seed, n)
            bm = _sensor_bitmaps(bins, case, n_words)
        st["eng"] = Engine(hbm_budget=8 * GB)
        d = bm.shape[0]
        st["d"], st["n_words"] = d, n_words
        if kind == "cooc":
            st["bm"] = bm
            st["out"] = torch.zeros((d, d), dtype=torch.int32, device=DEV)
            return st
        rng = np.random.default_rng(seed)
        cp, ci = _walk_sets(case, rng) if case["data"] == "sparse" else _occurring_sets(case, rng, bins)
        if case["api"] == "host":
            st["eng"].load_bitmaps(bm.cpu().numpy().view(np.uint64), n)
            st["cp"], st["ci"] = cp, ci
            return st
        st["bm"] = bm
        st["cp"] = torch.from_numpy(cp.view(np.int64)).to(DEV)
        st["ci"] = torch.from_numpy(ci.view(np.int32)).to(DEV)
        st["out"] = torch.zeros(case["n_cand"], dtype=torch.int32, device=DEV)
        return st
    if kind == "mine":
        rows = _sensor_items(_shuffled(_sensor_bins(case, case["model"], case["n_txn"]), seed), case, seed)
        st["ptr"] = np.arange(len(rows) + 1, dtype=np.uint64) * np.uint64(rows.shape[1])
        st["items"] = rows.reshape(-1)
        st["eng"] = Engine(hbm_budget=16 * GB)
        return st
    if kind == "anytime":
        bins = _shuffled(_sensor_bins(case, case["model"], case["n_txn"]), seed)
        bm = _sensor_bitmaps(bins, case, _words(case["n_txn"]))
        bm = bm[torch.tensor(np.random.default_rng(seed).permutation(len(bm)), device=DEV)]
        st["eng"] = Engine(hbm_budget=64 * GB)
        st["eng"].load_bitmaps(bm.cpu().numpy().view(np.uint64), case["n_txn"])
        return st
    if kind == "windows":
        rng = np.random.default_rng(case["model"])
        lens = np.exp(rng.uniform(np.log(case["len_lo"]), np.log(case["len_hi"]), case["n_win"])).astype(np.int64)
        n = 4 * case["len_hi"]
        stream = dict(sensors=21, bins=6, regimes=8, alpha=0.3, model=case["model"])
        rows = _sensor_items(_sensor_bins(stream, case["model"], n), stream, seed)
        st["ring"] = Ring(126, n)
        st["ring"].append(np.arange(n + 1, dtype=np.uint64) * np.uint64(21), rows.reshape(-1))
        ends = rng.integers(case["len_hi"], n + 1, case["n_win"])
        order = np.random.default_rng(seed).permutation(case["n_win"])
        st["starts"], st["lens"] = (ends - lens)[order], lens[order]
        st["floors"] = np.ceil(case["floor"] * st["lens"]).astype(np.int64)
        st["eng"] = Engine(hbm_budget=32 * GB)
        return st
    if kind in ("train", "score"):
        x, y, wt, p = _scorer(case, seed)
        st["eng"] = Engine(hbm_budget=GB)
        st["tr"] = tr = Trainer(st["eng"], in_dim=8, hidden=case["hidden"])
        for k, v in p.items():
            tr.p[k].copy_(torch.from_numpy(v))
            if k in tr.b16:
                tr.b16[k].copy_(torch.from_numpy(to_bf16_bits(v).view(np.int16)))
        st["x"], st["y"], st["wt"] = (torch.from_numpy(a).to(DEV) for a in (x, y, wt))
        return st
    st["vals"], st["anomaly"] = _stream(case, seed)
    st["eng"] = Engine(hbm_budget=8 * GB)
    return st


def run(st):
    case, eng = st["case"], st["eng"]
    kind = case["kind"]
    if kind == "support":
        if case["api"] == "host":
            return eng.support_batch(st["cp"], st["ci"]).view(np.int32)
        eng.support_batch_device(st["bm"].data_ptr(), st["d"], st["n_words"], st["n_words"], st["cp"].data_ptr(),
                                 st["ci"].data_ptr(), case["n_cand"], st["out"].data_ptr(),
                                 torch.cuda.current_stream().cuda_stream)
        return st["out"]
    if kind == "cooc":
        eng.cooccurrence_device(st["bm"].data_ptr(), st["d"], st["n_words"], st["n_words"], st["out"].data_ptr(),
                                stream=torch.cuda.current_stream().cuda_stream)
        return st["out"]
    if kind == "mine":
        res = eng.load_csr(st["ptr"], st["items"]).mine(max(1, int(math.ceil(case["floor"] * case["n_txn"]))),
                                                        order=case["order"])
        return {"ptr": res.ptr.view(np.int64), "items": res.items.view(np.int32), "support": res.support.view(np.int32)}
    if kind == "anytime":
        res = eng.mine(int(math.ceil(case["floor"] * case["n_txn"])))
        return {"ptr": res.ptr.view(np.int64), "items": res.items.view(np.int32), "support": res.support.view(np.int32)}
    if kind == "windows":
        res = st["ring"].mine_windows(eng, st["starts"], st["lens"], st["floors"])
        return {"offset": res.offset.view(np.int64), "masks": res.masks.view(np.int64),
                "support": res.support.view(np.int32), "status": res.status}
    if kind == "train":
        loss, grads = st["tr"].gradients(st["x"], st["y"], st["wt"])
        return {"loss": loss, "grads": grads}
    if kind == "score":
        return st["tr"].forward(st["x"])
    if case["online"]:
        items, labels, edges = eng.transactionize_online(st["vals"], case["window"], case["stride"], case["bins"],
                                                         anomaly=st["anomaly"])
    else:
        items, labels, edges = eng.transactionize(st["vals"], case["window"], case["stride"], case["bins"],
                                                  anomaly=st["anomaly"])
    return {"items": items, "labels": labels, "edges": edges}


def work(case):
    """Inputs read once, outputs written once.  Bitmap work counts no floating-point operations, except
    co-occurrence, which is a product of the 0/1 matrix with itself (its upper triangle)."""
    kind = case["kind"]
    if kind in ("support", "cooc"):
        d = _items_of(case)
        bits = d * _words(case["n_txn"]) * 8
        if kind == "cooc":
            return {"bytes": bits + 4 * d * d, "flops": float(d) * (d + 1) * case["n_txn"]}
        k = (case["kmin"] + case["kmax"]) / 2
        return {"bytes": bits + case["n_cand"] * (8 + 4 * k + 4), "flops": 0}
    if kind == "mine":
        return {"bytes": case["n_txn"] * (8 + 4 * case["sensors"]), "flops": 0}
    if kind == "anytime":
        return {"bytes": _items_of(case) * _words(case["n_txn"]) * 8, "flops": 0}
    if kind == "windows":
        mean = (case["len_hi"] - case["len_lo"]) / math.log(case["len_hi"] / case["len_lo"])
        return {"bytes": case["n_win"] * mean * 126 / 8, "flops": 0}
    if kind in ("train", "score"):
        n, h = case["rows"], case["hidden"]
        params = h * 8 + h * h + 3 * h + 1
        if kind == "score":
            return {"bytes": 4 * n * (8 + 1) + 2 * params, "flops": 2.0 * n * (8 * h + h * h + h)}
        return {"bytes": 4 * n * (8 + 2) + 6 * params, "flops": 6.0 * n * (8 * h + h * h + h)}
    n_win = (case["rows"] - case["window"]) // case["stride"] + 1
    out = n_win * 4 * (case["sensors"] + 1) + (n_win * case["sensors"] * (case["bins"] + 1) * 8 if case["online"] else 0)
    return {"bytes": case["rows"] * (8 * case["sensors"] + 4) + out, "flops": 0}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("train", "score"):
        x, y, wt, p = _scorer(case, seed)
        x, y, wt = (torch.from_numpy(a).to(DEV, torch.float64) for a in (x, y, wt))
        p = {k: torch.from_numpy(v).to(DEV, torch.float64) for k, v in p.items()}
        z1 = x @ p["W1"].T + p["b1"]
        h1 = z1.clamp(min=0)
        z2 = h1 @ p["W2"].T + p["b2"]
        h2 = z2.clamp(min=0)
        prob = torch.sigmoid(h2 @ p["w3"] + p["b3"])
        if kind == "score":
            return prob
        q = prob.clamp(1e-7, 1 - 1e-7)
        loss = -(wt * (y * torch.log(q) + (1 - y) * torch.log(1 - q))).mean().reshape(1)
        g3 = wt * (prob - y) / len(y)
        g2 = g3[:, None] * p["w3"] * (z2 > 0)
        g1 = (g2 @ p["W2"]) * (z1 > 0)
        return {"loss": loss, "grads": {"W1": g1.T @ x, "b1": g1.sum(0), "W2": g2.T @ h1, "b2": g2.sum(0),
                                        "w3": h2.T @ g3, "b3": g3.sum().reshape(1)}}
    if kind == "transact" and not case["online"]:
        vals, _ = _stream(case, seed)
        q = np.quantile(vals, np.linspace(0, 1, case["bins"] + 1), axis=0)
        return {"items": None, "labels": None, "edges": [np.unique(q[:, s]) for s in range(case["sensors"])]}
    return None
