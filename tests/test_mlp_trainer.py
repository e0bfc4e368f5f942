"""Host logic of the scorer's trainer on the CPU, with a fake engine: fit() asks for the device status once an
epoch and raises when a forward or backward pass gave up on a wait."""
import pytest

torch = pytest.importorskip("torch")

from sgfim import _lib as L  # noqa: E402
from sgfim.engine import SgfimError  # noqa: E402
from sgfim.mlp import Trainer  # noqa: E402


class FakeEngine:
    """Counts the status calls; the one of epoch `bad` reports a wait that ran out."""

    def __init__(self, bad=None):
        self.bad, self.asked = bad, 0

    def device_status(self, stream=0):
        self.asked += 1
        return L.EDEVICE if self.asked - 1 == self.bad else 0


def _trainer(engine):
    t = Trainer.__new__(Trainer)
    t.torch, t.eng, t.dev = torch, engine, torch.device("cpu")
    t._stream = lambda: 0
    t.seen = []
    t.step = lambda X, Y, WT=None, lr=1e-3: (t.seen.append(len(X)), torch.ones(1))[1]
    return t


def test_fit_checks_the_device_every_epoch():
    t = _trainer(FakeEngine())
    hist = t.fit(torch.zeros(10, 8), torch.tensor([0.0, 1.0] * 5), epochs=3, batch=4)
    assert hist == [1.0, 1.0, 1.0] and t.seen == [4, 4, 2] * 3
    assert t.eng.asked == 3


@pytest.mark.parametrize("bad", [0, 2])
def test_fit_raises_when_a_wait_ran_out(bad):
    t = _trainer(FakeEngine(bad))
    with pytest.raises(SgfimError) as e:
        t.fit(torch.zeros(10, 8), torch.tensor([0.0, 1.0] * 5), epochs=3, batch=4)
    assert e.value.code == L.EDEVICE
    assert len(t.seen) == 3 * (bad + 1)     # no step after the epoch that failed


def test_gradients_clear_entries_that_a_caller_replaced():
    """g[k] may be the caller's own tensor: every entry is cleared before the backward adds to it."""
    class Adds:
        def mlp_backward(self, *a):
            for t in self.g.values():
                t += 1.0
    eng = Adds()
    t = Trainer.__new__(Trainer)
    t.torch, t.eng, t.dev, t.in_dim, t.hidden = torch, eng, torch.device("cpu"), 8, 32
    t._stream = lambda: 0
    t.forward = lambda X, keep=False: (torch.zeros(len(X)),) * 3
    t.p = {"W1": torch.zeros(32, 8), "b1": torch.zeros(32), "W2": torch.zeros(32, 32), "b2": torch.zeros(32),
           "w3": torch.zeros(32), "b3": torch.zeros(1)}
    t.b16 = {"W2": torch.zeros(32, 32, dtype=torch.int16), "w3": torch.zeros(32, dtype=torch.int16)}
    t._alloc_gradients()
    eng.g = t.g
    mine = torch.full((32, 8), 7.0)
    t.g["W1"] = mine
    for _ in range(3):
        _, g = t.gradients(torch.zeros(4, 8), torch.zeros(4))
    assert g["W1"] is mine
    for k in t.p:
        assert g[k].shape == t.p[k].shape and bool((g[k] == 1.0).all()), k
