"""The scorer's tensor-core forward and its backward at the edges of their tiles: hidden widths of one
and several K chunks and column blocks, row counts around the 128-row tile and the 32-row batch, wide
inputs, pointers that forbid 16-byte accesses, infinite activations and weights.

Tolerances: every product is exact in fp32 and each sum has at most 256 + 64 terms, so a
pre-activation is within 400 * 2^-24 * sum |terms| of the float64 value (2.4e-5 of it); probabilities
move by at most a quarter of the logit's error.  Gradients: sums over n rows of such values, 1e-4 of
the largest entry at the sizes here."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _net(torch, n, F, H, seed):
    from sgfim.mlp import from_bf16_bits, to_bf16_bits
    rng = np.random.default_rng(seed)
    r = lambda *s: rng.uniform(-1, 1, s)  # noqa: E731
    bf = lambda a: from_bf16_bits(to_bf16_bits(a))  # noqa: E731
    w = {"X": rng.random((n, F)).astype(np.float32), "W1": bf(r(H, F) * np.sqrt(3 / F)),
         "b1": r(H).astype(np.float32) * 0.1, "W2": bf(r(H, H) * np.sqrt(3 / H)), "b2": r(H).astype(np.float32) * 0.1,
         "w3": bf(r(H) * np.sqrt(3 / H)), "b3": r(1).astype(np.float32),
         "Y": (rng.random(n) < 0.4).astype(np.float32), "WT": rng.uniform(0.5, 2, n).astype(np.float32)}
    return w


def _run(torch, eng, w, shift=0, backward=True):
    from sgfim.mlp import to_bf16_bits
    n, F = w["X"].shape
    H = len(w["b1"])
    keep = []

    def dev(a, dtype=torch.float32):   # shift > 0: the data start at an address that is not a multiple of 16
        t = torch.zeros(a.size + 8, dtype=dtype, device="cuda")
        t[shift:shift + a.size] = torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).to("cuda")
        keep.append(t)
        return t[shift:shift + a.size]
    f = {k: dev(w[k]) for k in ("X", "b1", "b2", "b3", "Y", "WT")}
    b = {k: dev(to_bf16_bits(w[k]).view(np.int16), torch.int16) for k in ("W1", "W2", "w3")}
    Z1, Z2, P = dev(np.zeros(n * H, np.float32)), dev(np.zeros(n * H, np.float32)), dev(np.zeros(n, np.float32))
    st = torch.cuda.current_stream().cuda_stream
    eng.mlp_forward(f["X"].data_ptr(), n, F, H, b["W1"].data_ptr(), f["b1"].data_ptr(), b["W2"].data_ptr(),
                    f["b2"].data_ptr(), b["w3"].data_ptr(), f["b3"].data_ptr(), Z1.data_ptr(), Z2.data_ptr(),
                    P.data_ptr(), st)
    out = {"Z1": Z1, "Z2": Z2, "P": P}
    if backward:
        g = {k: dev(np.zeros(s, np.float32)) for k, s in (("W1", H * F), ("b1", H), ("W2", H * H), ("b2", H), ("w3", H),
                                                          ("b3", 1), ("loss", 1))}
        eng.mlp_backward(f["X"].data_ptr(), n, F, H, b["W2"].data_ptr(), b["w3"].data_ptr(), Z1.data_ptr(),
                         Z2.data_ptr(), P.data_ptr(), f["Y"].data_ptr(), f["WT"].data_ptr(), 1.0 / n,
                         g["W1"].data_ptr(), g["b1"].data_ptr(), g["W2"].data_ptr(), g["b2"].data_ptr(),
                         g["w3"].data_ptr(), g["b3"].data_ptr(), g["loss"].data_ptr(), st)
        out.update(g)
    assert eng.device_status(st) == 0
    return {k: v.cpu().numpy().astype(np.float64) for k, v in out.items()}


def _ref(w):
    from sgfim.mlp import from_bf16_bits, to_bf16_bits
    w = {k: (from_bf16_bits(to_bf16_bits(v)) if k in ("W1", "W2", "w3") else v).astype(np.float64)
         for k, v in w.items()}   # the weights as the kernels see them
    n = len(w["X"])
    z1 = w["X"] @ w["W1"].T + w["b1"]
    h1 = np.maximum(z1, 0)
    z2 = h1 @ w["W2"].T + w["b2"]
    p = 1 / (1 + np.exp(-(np.maximum(z2, 0) @ w["w3"] + w["b3"])))
    q = np.clip(p, 1e-7, 1 - 1e-7)
    g3 = w["WT"] * (p - w["Y"]) / n
    g2 = g3[:, None] * w["w3"] * (z2 > 0)
    g1 = (g2 @ w["W2"]) * (z1 > 0)
    return {"Z1": z1, "Z2": z2, "P": p, "loss": -(w["WT"] * (w["Y"] * np.log(q) + (1 - w["Y"]) * np.log(1 - q))).mean(),
            "W1": g1.T @ w["X"], "b1": g1.sum(0), "W2": g2.T @ h1, "b2": g2.sum(0),
            "w3": np.maximum(z2, 0).T @ g3, "b3": g3.sum()}


@pytest.mark.parametrize("n,F,H,shift", [(1, 8, 32, 0), (127, 1, 64, 0), (129, 8, 96, 1), (300, 9, 128, 0),
                                         (4097, 8, 128, 3), (257, 64, 160, 0), (130, 64, 256, 0), (1000, 8, 256, 2)])
def test_forward_backward_shapes(engine, n, F, H, shift):
    torch = pytest.importorskip("torch")
    w = _net(torch, n, F, H, n)
    got, want = _run(torch, engine, w, shift), _ref(w)
    scale = max(1.0, np.abs(want["Z2"]).max())
    for k in ("Z1", "Z2"):
        assert np.abs(got[k].reshape(want[k].shape) - want[k]).max() < 2.4e-5 * 4 * scale, k
    assert np.abs(got["P"] - want["P"]).max() < 2.4e-5 * 4
    assert abs(got["loss"][0] - want["loss"]) < 1e-4
    for k in ("W1", "b1", "W2", "b2", "w3", "b3"):
        ref = np.asarray(want[k]).reshape(-1)
        # a pre-activation within its error of zero may take the other side of the ReLU: one row's share
        assert np.abs(got[k] - ref).max() <= 1e-4 * np.abs(ref).max() + 1e-7, k


def test_forward_infinite_values(engine):
    """An infinite activation and an infinite weight give what the plain sums give."""
    torch = pytest.importorskip("torch")
    w = _net(torch, 200, 8, 64, 3)
    w["X"][7, 2] = np.inf
    w["W1"][:, 2] = np.abs(w["W1"][:, 2]) + 0.5      # h1 of row 7 is +inf in every unit
    w["W2"] = np.where(w["W2"] == 0, np.float32(0.5), w["W2"])
    w["W2"][5] = np.abs(w["W2"][5])                  # unit 5 of layer 2 sums infinities of one sign
    got = _run(torch, engine, w, backward=False)
    z2 = got["Z2"].reshape(200, 64)
    assert z2[7, 5] == np.inf
    mixed = (w["W2"] > 0).any(1) & (w["W2"] < 0).any(1)
    assert np.isnan(z2[7, mixed]).all()
    rest = np.arange(200) != 7
    want = _ref({k: (v[rest] if k in ("X", "Y", "WT") else v) for k, v in w.items()})
    assert np.abs(z2[rest] - want["Z2"]).max() < 1e-4 * max(1, np.abs(want["Z2"]).max())
    w = _net(torch, 200, 8, 64, 4)
    w["W1"] = np.abs(w["W1"])
    w["b1"] = np.abs(w["b1"]) + np.float32(0.1)      # every activation is positive
    w["W2"][9, 3] = np.inf
    got = _run(torch, engine, w, backward=False)
    z2 = got["Z2"].reshape(200, 64)
    assert (z2[:, 9] == np.inf).all()
    fin = np.delete(np.arange(64), 9)
    w["W2"][9, 3] = 0
    assert np.abs(z2[:, fin] - _ref(w)["Z2"][:, fin]).max() < 1e-4 * np.abs(_ref(w)["Z2"]).max()


@pytest.mark.parametrize("n,H", [(1, 32), (127, 64), (128, 96), (129, 128), (256, 32), (5000, 128)])
def test_eight_inputs_shapes(engine, n, H):
    """Eight aligned inputs a row are fetched a tile ahead: inputs of both signs and of magnitudes
    from 1e-30 to 1e3."""
    torch = pytest.importorskip("torch")
    w = _net(torch, n, 8, H, n + H)
    rng = np.random.default_rng(n)
    w["X"] = (rng.uniform(-1, 1, (n, 8)) * 10.0 ** rng.choice([-30, -3, 0, 0, 0, 3], (n, 8))).astype(np.float32)
    got, want = _run(torch, engine, w, backward=False), _ref(w)
    # sums of at most 8 + H exact products: 400 * 2^-24 of the terms' magnitudes
    t1 = np.abs(w["X"].astype(np.float64)) @ np.abs(w["W1"].astype(np.float64)).T + np.abs(w["b1"])
    t2 = t1 @ np.abs(w["W2"].astype(np.float64)).T + np.abs(w["b2"])
    assert (np.abs(got["Z1"].reshape(n, H) - want["Z1"]) <= 2.4e-5 * t1).all()
    assert (np.abs(got["Z2"].reshape(n, H) - want["Z2"]) <= 2.4e-5 * t2).all()
    t3 = t2 @ np.abs(w["w3"].astype(np.float64)) + np.abs(w["b3"])
    assert (np.abs(got["P"] - want["P"]) <= 2.4e-5 * t3 / 4 + 1e-7).all()


def test_eight_inputs_infinite_values(engine):
    """Infinite and NaN inputs and an infinite layer-1 weight give what the plain sums give."""
    torch = pytest.importorskip("torch")
    w = _net(torch, 300, 8, 128, 9)
    w["W1"] = np.where(w["W1"] == 0, np.float32(0.5), w["W1"])
    w["X"][3, 1], w["X"][4, 6], w["X"][131, 0] = np.inf, -np.inf, np.nan
    z1 = _run(torch, engine, w, backward=False)["Z1"].reshape(300, 128)
    assert (z1[3] == np.inf * np.sign(w["W1"][:, 1])).all() and (z1[4] == -np.inf * np.sign(w["W1"][:, 6])).all()
    assert np.isnan(z1[131]).all()
    rest = np.delete(np.arange(300), [3, 4, 131])
    want = _ref({k: (v[rest] if k in ("X", "Y", "WT") else v) for k, v in w.items()})["Z1"]
    assert np.abs(z1[rest] - want).max() < 1e-4 * np.abs(want).max()
    w = _net(torch, 300, 8, 128, 10)
    w["X"] = np.abs(w["X"]) + np.float32(0.01)
    w["W1"][17, 5] = -np.inf
    got = _run(torch, engine, w, backward=False)
    z1, z2 = got["Z1"].reshape(300, 128), got["Z2"].reshape(300, 128)
    assert (z1[:, 17] == -np.inf).all()
    fin = np.delete(np.arange(128), 17)
    w["W1"][17] = 0
    w["b1"][17] = -1                 # its activation is zero either way
    want = _ref(w)
    assert np.abs(z1[:, fin] - want["Z1"][:, fin]).max() < 1e-4 * np.abs(want["Z1"]).max()
    assert np.abs(z2 - want["Z2"]).max() < 1e-4 * np.abs(want["Z2"]).max()
