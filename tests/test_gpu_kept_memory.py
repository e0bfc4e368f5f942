"""What a handle keeps on the device between calls is bounded by its memory budget: the buffers of
transactionisation and loading go back when they exceed a sixteenth of it, and an AUTO support call takes the
tables of the pair groups only up to an eighth.  Free device memory is read before and after a call whose
kernels another handle has loaded before; 8 MB of slack are the allocator's granules."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _kept(call, budget):
    """Device memory that a fresh handle with this budget still holds after call(handle), less what it held before."""
    import torch
    from sgfim.engine import Engine
    with Engine(hbm_budget=1 << 30) as warm:
        call(warm)
    torch.cuda.synchronize()
    with Engine(hbm_budget=budget) as eng:
        before = torch.cuda.mem_get_info()[0]
        out = call(eng)
        torch.cuda.synchronize()
        return before - torch.cuda.mem_get_info()[0], out


@pytest.mark.parametrize("online", [False, True])
def test_transactionise_gives_large_buffers_back(online):
    vals = np.random.default_rng(1).normal(size=(200_000, 20))

    def call(eng):
        f = eng.transactionize_online if online else eng.transactionize
        return f(vals, 30, 15, 5)[0]
    small, a = _kept(call, 64 * MB)
    large, b = _kept(call, 16 << 30)
    assert np.array_equal(a, b)
    assert small <= 8 * MB, small          # 32 MB of rows alone
    assert large >= 24 * MB, large         # and kept where the budget allows


def test_load_gives_large_buffers_back():
    n = 400_000
    ptr = np.arange(n + 1, dtype=np.uint64) * np.uint64(8)
    items = np.random.default_rng(2).integers(0, 40, n * 8).astype(np.uint32)
    bitmaps = 40 * ((n + 63) // 64) * 8
    kept, _ = _kept(lambda eng: eng.load_csr(ptr, items), 64 * MB)
    assert kept <= bitmaps + 8 * MB, kept  # 16 MB of the CSR on its way


def test_auto_pair_groups_stay_within_the_budget():
    import torch
    d, n_txn, n = 300, 262_144, 500_000
    rng = np.random.default_rng(3)
    bm = torch.from_numpy(np.packbits(rng.random((d, n_txn)) < 0.05, axis=1, bitorder="little").view(np.int64)).cuda()
    ci = rng.integers(0, d, n * 5).astype(np.uint32)
    cp = np.arange(n + 1, dtype=np.uint64) * np.uint64(5)
    tp, ti = torch.from_numpy(cp.view(np.int64)).cuda(), torch.from_numpy(ci.view(np.int32)).cuda()
    outs = [torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2)]

    def call(out):
        def f(eng):
            eng.support_batch_device(bm.data_ptr(), d, n_txn // 64, n_txn // 64, tp.data_ptr(), ti.data_ptr(), n,
                                     out.data_ptr(), torch.cuda.current_stream().cuda_stream)
        return f
    small, _ = _kept(call(outs[0]), 128 * MB)
    large, _ = _kept(call(outs[1]), 16 << 30)
    assert torch.equal(outs[0], outs[1])
    assert small <= 24 * n + 8 * MB, small      # the lane kernels' 24 bytes a candidate
    assert large >= 80 * n, large
