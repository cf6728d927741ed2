"""Kernels of a search that take their places while their predecessor drains, against the same search captured into a graph,
whose launches wait for one another: the same results, with searches of different shapes in a row on one scratch and no
wait between them, and no longer times where a kernel depends on the SMs' division of shared memory and L1."""
import ctypes

import numpy as np
import pytest

import helpers as H
from oracle import flat_oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def captured(fm, side, a):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        fm.abi.check_op(fm.lib().b200f_search(ctypes.byref(a)), "captured search")
    return graph


@pytest.mark.parametrize("nq,nb,k", [(148, 32_000, 10), (1000, 100_000, 40)])
def test_equal_rows_are_selected_from_l1(fm, res, nq, nb, k):
    # rows of equal keys, read several times by the selection: 190 against 130 us (148 queries), 12 against 10 ms where it
    # kept the distance kernel's division
    from test_gpu_ops import Stored
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        st = Stored(fm, np.tile(H.gaussian(1, 64, 1), (nb, 1)), 2)
        xq = torch.from_numpy(H.gaussian(nq, 64, 2)).cuda()
        D = torch.empty((nq, k), dtype=torch.float32, device="cuda:0")
        I = torch.empty((nq, k), dtype=torch.int64, device="cuda:0")
        a = st.args(fm, xq, O.METRIC_L2, k, 2, D, I)
        a.stream = side.cuda_stream
        eager = lambda: fm.abi.check_op(fm.lib().b200f_search(ctypes.byref(a)), "search")
        eager()
        side.synchronize()
        graph = captured(fm, side, a)
        best = []
        for run in (eager, graph.replay):
            t = []
            for _ in range(10):
                t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                t0.record(side)
                run()
                t1.record(side)
                side.synchronize()
                t.append(1e3 * t0.elapsed_time(t1))
            best.append(min(t))
    assert (I.cpu().numpy() == np.arange(k)).all()
    assert best[0] <= 1.1 * best[1] + 10, best


def test_searches_in_a_row_on_one_scratch(fm, res):
    # no wait between the searches: what one leaves in the scratch, and its last kernels, meet the next one's first
    from test_gpu_ops import Stored
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        shapes = []
        for storage, metric, nb, d, seed in ((2, O.METRIC_L2, 70_000, 48, 1), (0, O.METRIC_INNER_PRODUCT, 40_000, 100, 2), (1, O.METRIC_L2, 600_000, 16, 3)):
            xb = H.gaussian(nb, d, seed)
            xb[nb // 2:nb // 2 + 9000] = xb[3]   # the queries near these are redone
            st = Stored(fm, xb, storage)
            for nq, k, path in ((1, 10, 0), (4, 32, 0), (8, 200, 0), (20, 40, 2), (130, 10, 2), (300, 300, 2), (9, 2000, 2)):
                xq = H.gaussian(nq, d, 10 * seed + nq)
                xq[nq // 2] = xb[3] + 0.01
                xq = torch.from_numpy(xq).cuda()
                shapes.append((st, xq, metric, k, path))
        calls, keep = [], []
        for st, xq, metric, k, path in shapes:
            D = torch.empty((len(xq), k), dtype=torch.float32, device="cuda:0")
            I = torch.empty((len(xq), k), dtype=torch.int64, device="cuda:0")
            a = st.args(fm, xq, metric, k, path, D, I)
            a.stream = side.cuda_stream
            keep.append((st.scratch, st.status))
            calls.append((a, D, I))
        scratch = torch.empty(max(a.scratch_bytes for a, _, _ in calls), dtype=torch.uint8, device="cuda:0")
        for a, _, _ in calls:
            a.scratch, a.scratch_bytes = scratch.data_ptr(), scratch.numel()
        search = lambda a: fm.abi.check_op(fm.lib().b200f_search(ctypes.byref(a)), "search")
        for a, _, _ in calls:
            search(a)
        side.synchronize()
        want = []
        for a, D, I in calls:
            graph = captured(fm, side, a)
            graph.replay()
            side.synchronize()
            want.append((D.clone(), I.clone()))
        order = list(range(len(calls)))
        for rounds in range(6):
            np.random.default_rng(rounds).shuffle(order)
            for i in order:
                calls[i][1].fill_(0)
                calls[i][2].fill_(-7)
            for i in order:
                search(calls[i][0])
            side.synchronize()
            for i in order:
                assert torch.equal(calls[i][1], want[i][0]) and torch.equal(calls[i][2], want[i][1]), (rounds, i)
        assert all(int(words[0]) == 0 for _, words in keep)
        assert sum(int(words[1]) > 0 for _, words in keep) >= 3   # redos were among them
