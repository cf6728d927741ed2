"""A search's status words where the host paths keep them, in pinned memory that the kernels write: the number of redone
queries comes once a search, and an error that has been reported is not reported again."""
import ctypes

import numpy as np
import pytest

import helpers as H
from oracle import flat_oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


# lists, one matrix chunk, several chunks, streaming scans (lists and candidates)
@pytest.mark.parametrize("storage,nq,nb,k", [(1, 1000, 70_000, 10), (2, 1000, 70_000, 100), (0, 4000, 70_000, 40),
                                             (2, 4, 600_000, 32), (1, 3, 70_000, 200)])
def test_redone_queries(fm, res, storage, nq, nb, k):
    from test_gpu_ops import Stored
    # equal rows: every one passes a threshold, no buffer holds them, all queries are redone
    st = Stored(fm, np.tile(H.gaussian(1, 16, 1), (nb, 1)), storage)
    xq = torch.from_numpy(H.gaussian(nq, 16, 2)).cuda()
    D = torch.empty((nq, k), dtype=torch.float32, device="cuda:0")
    I = torch.empty((nq, k), dtype=torch.int64, device="cuda:0")
    a = st.args(fm, xq, O.METRIC_L2, k, 0, D, I)
    pinned = torch.full((4,), -1, dtype=torch.int32).pin_memory()
    times = []
    for words in (st.status, pinned):
        a.status = words.data_ptr()
        best = float("inf")
        for _ in range(5):
            t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            t0.record()
            fm.abi.check_op(fm.lib().b200f_search(ctypes.byref(a)), "search")
            t1.record()
            torch.cuda.synchronize()
            assert words.tolist() == [0, nq, 0, 0]
            best = min(best, t0.elapsed_time(t1))
        times.append(best)
    assert (I.cpu().numpy() == np.arange(k)).all()
    # an atomic a redone row across PCIe took 0.9 us each; two writes a search take none that shows
    assert times[1] <= times[0] + 0.2, times


def test_an_error_is_reported_once(fm, res):
    idx = fm.B200IndexFlat(res, 32, O.METRIC_L2, 1)
    idx.add(H.gaussian(5000, 32, 1))
    xq = H.gaussian(1, 32, 2)
    for _ in range(3):   # the third is replayed from a graph
        D, I = idx.search(xq, 5)
    fm.abi.check(fm.lib().b200f_index_debug_wait_expiry(idx._h, 2_000_000), "debug_wait_expiry")
    with pytest.raises(fm.B200Error):
        idx.synchronize()
    assert idx.last_device_status == 1
    idx.synchronize()
    D2, I2 = idx.search(xq, 5)
    assert np.array_equal(D, D2) and np.array_equal(I, I2)
    idx.synchronize()
    idx.close()
