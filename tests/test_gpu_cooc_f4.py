"""Co-occurrence with fp4 operands against the exact integer product, at the edges of its tiles (128 and 256
rows), its steps (256 transactions) and its runs of 2^20 transactions; full rows show that sums of a whole
run stay exact in fp32."""
import numpy as np
import pytest

from sgfim import _lib as L

pytestmark = pytest.mark.gpu


def _exact(bm):
    bits = np.unpackbits(bm.view(np.uint8), axis=1, bitorder="little")
    out = np.zeros((len(bm), len(bm)), np.float64)
    for a in range(0, bits.shape[1], 1 << 16):      # integer products, exact in float64
        x = bits[:, a:a + (1 << 16)].astype(np.float32)
        out += (x @ x.T).astype(np.float64)         # at most 2^16 per product: exact in fp32
    return out.astype(np.uint32)


def _run(engine, bm, kind):
    import torch
    words = (bm.shape[1] + 1) & ~1
    pad = np.zeros((len(bm), words), np.uint64)
    pad[:, :bm.shape[1]] = bm
    t = torch.from_numpy(pad.view(np.int64)).cuda()
    out = torch.full((len(bm), len(bm)), 7, dtype=torch.int32, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    engine.cooccurrence_device(t.data_ptr(), len(bm), bm.shape[1], words, out.data_ptr(), kind, st)
    assert engine.device_status(st) == 0
    return out.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("d,words,dens", [(1, 1, 0.5), (2, 4, 0.5), (126, 1024, 0.17), (127, 5, 0.3), (128, 63, 0.3),
                                          (129, 64, 0.1), (255, 7, 0.6), (256, 130, 0.2), (257, 3, 0.9),
                                          (640, 400, 0.1), (1025, 90, 0.1)])
def test_cooc_f4_random(engine, d, words, dens):
    rng = np.random.default_rng(d)
    bm = np.packbits(rng.random((d, words * 64)) < dens, axis=1, bitorder="little").view(np.uint64)
    want = _exact(bm)
    assert np.array_equal(_run(engine, bm, L.COOC_TC_F4), want)
    assert np.array_equal(_run(engine, bm, L.COOC_AUTO), want)


@pytest.mark.parametrize("d,n_txn", [(3, (1 << 20) + 64), (300, 1 << 20), (1500, 1 << 20), (130, (1 << 21) + 4096)])
def test_cooc_f4_full_rows(engine, d, n_txn):
    bm = np.full((d, n_txn // 64), ~np.uint64(0))
    bm[d // 2, ::3] = 0x5555555555555555
    got = _run(engine, bm, L.COOC_TC_F4)
    half = n_txn - 32 * len(range(0, n_txn // 64, 3))
    want = np.full((d, d), n_txn, np.uint32)
    want[d // 2, :] = half
    want[:, d // 2] = half
    assert np.array_equal(got, want)


@pytest.mark.parametrize("d,words", [(1024, 512), (1024, 514), (300, 512), (257, 966), (1051, 78), (1400, 128), (700, 10)])
def test_cooc_f4_short_last_run(engine, d, words):
    """Shapes whose last run of transactions is short and dealt in whole tiles."""
    rng = np.random.default_rng(d + words)
    bm = np.packbits(rng.random((d, words * 64)) < 0.2, axis=1, bitorder="little").view(np.uint64)
    assert np.array_equal(_run(engine, bm, L.COOC_AUTO), _exact(bm))


@pytest.mark.parametrize("kind", [L.COOC_TC_F8, L.COOC_TC_F8_256, L.COOC_TC_F4])
@pytest.mark.parametrize("d,words", [(256, 16384), (400, 4688)])
def test_cooc_tensor_kernels_repeat_exactly(engine, kind, d, words):
    """Thousands of calls of a tensor-core kernel agree with the popcount kernel: a ring slot that is refilled before
    its bits are used shows in one call of a few thousand, on diagonal blocks first."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(d)
    bm = torch.randint(-2**63, 2**63 - 1, (d, words), generator=g, device="cuda", dtype=torch.int64)
    bm &= torch.randint(-2**63, 2**63 - 1, (d, words), generator=g, device="cuda", dtype=torch.int64)
    st = torch.cuda.current_stream().cuda_stream
    want, out = (torch.zeros((d, d), dtype=torch.int32, device="cuda") for _ in range(2))
    engine.cooccurrence_device(bm.data_ptr(), d, words, words, want.data_ptr(), L.COOC_POPC, st)
    bad = torch.zeros((), dtype=torch.int64, device="cuda")
    for _ in range(8000):
        engine.cooccurrence_device(bm.data_ptr(), d, words, words, out.data_ptr(), kind, st)
        bad += (out != want).any()
    assert engine.device_status(st) == 0
    assert int(bad) == 0
