"""Small searches from host buffers, replayed from a graph that fetches the queries by a kernel or (more than 64 KB) copies
them: query blocks that are no whole number of the kernel's 256-byte pieces, and wide ones, which must not wait for one
warp's reads across PCIe."""
import time

import numpy as np
import pytest

import helpers as H
from oracle import flat_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d", [(1, 1), (1, 63), (1, 65), (8, 37), (3, 129), (1, 1025), (7, 1537), (8, 2047), (8, 2048), (8, 2049)])
def test_replay_equals_plain(fm, res, n, d):
    xb = H.uniform_pm1(3000, d, 1)
    idx = fm.B200IndexFlat(res, d, O.METRIC_L2, 0)
    plain = fm.B200IndexFlat(res, d, O.METRIC_L2, 0)
    plain.set_use_graphs(False)
    idx.add(xb)
    plain.add(xb)
    for rep in range(4):   # the second call captures, the others are replayed
        xq = H.uniform_pm1(n, d, 10 + rep)
        D, I = idx.search(xq, 5)
        Dp, Ip = plain.search(xq, 5)
        assert np.array_equal(I, Ip) and np.array_equal(D, Dp)
    idx.close()
    plain.close()


@pytest.mark.parametrize("d", [8192, 16384])
def test_wide_queries_are_not_slower(fm, res, d):
    xb = H.uniform_pm1(2000, d, 1)
    idx = fm.B200IndexFlat(res, d, O.METRIC_L2, 1)
    idx.add(xb)
    xq = [H.uniform_pm1(1, d, 10 + i) for i in range(8)]
    best = []
    for graphs in (False, True):
        idx.set_use_graphs(graphs)
        t = []
        for i in range(200):
            t0 = time.perf_counter()
            idx.search(xq[i % 8], 5)
            t.append(time.perf_counter() - t0)
        best.append(1e6 * np.median(t))
    # a warp alone took 1.2 us for every 2 KB: 20 us at d = 8192, 40 at 16384
    assert best[1] <= best[0] + 2, best
    idx.close()
