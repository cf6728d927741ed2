"""The distance GEMM that keeps the query block in shared memory (more than 128 queries, narrow rows): edges of its
k-blocks (64 columns, norm columns in a block of their own), of its tiles (256 rows of X, halves of 512) and of
its query blocks, the widths where the general kernel takes over, and ranges that change their query block."""
import ctypes

import numpy as np
import pytest
import torch

import helpers as H
from oracle import flat_oracle as O
from test_gpu_ops import Stored, cur_stream, vp

pytestmark = pytest.mark.gpu

# fp32 rows: two planes of up to three blocks, 16-bit rows: up to six; L2 adds eight norm columns
WIDTHS = {0: (8, 56, 64, 65, 128, 184, 185, 192, 193), 1: (63, 128, 376, 384, 385), 2: (16, 64, 320, 376, 377)}


@pytest.mark.parametrize("storage,d", [(s, d) for s, ds in WIDTHS.items() for d in ds])
@pytest.mark.parametrize("metric", [O.METRIC_L2, O.METRIC_INNER_PRODUCT])
@pytest.mark.parametrize("nq,nb", [(129, 1), (256, 256), (257, 769), (600, 40_001)])
def test_matrix(fm, res, storage, metric, d, nq, nb):
    xb = H.uniform_pm1(nb, d, 99)
    xq = H.uniform_pm1(nq, d, 77)
    st = Stored(fm, xb, storage)
    xq_dev = torch.from_numpy(xq).cuda()
    out = torch.full((nq, nb), float("nan"), dtype=torch.float32, device="cuda:0")
    a = st.args(fm, xq_dev, metric, 1, 2)
    if storage == 0:   # two fp16 planes of 2^6 x
        fm.abi.check_op(fm.lib().b200f_store_rows_fp32(vp(st.rows), st.pitch, nb, d, vp(st.rows), st.pitch, vp(st.planes),
                                                       st.ppitch, nb * st.ppitch, 1, 6, None, None, 1, cur_stream()), "planes")
        a.plane_format, a.plane_scale_log2 = 1, 6
    fm.abi.check_op(fm.lib().b200f_pairwise(ctypes.byref(a), vp(out), nb), "pairwise")
    torch.cuda.synchronize()
    assert int(st.status[0]) == 0
    xb_eff, xq_eff = H.effective_operands(storage, True, xb, xq)
    want = torch.from_numpy(xq_eff).cuda().double() @ torch.from_numpy(xb_eff).cuda().double().T
    if metric == O.METRIC_L2:
        want = ((xq.astype(np.float64) ** 2).sum(1)[:, None] + (xb_eff.astype(np.float64) ** 2).sum(1)[None]) - 2 * want.cpu().numpy()
        want = torch.from_numpy(want).cuda()
    # fp32 sums of at most 400 products and (fp32 rows) 2^-22 left out of each
    scale = float(want.abs().max())
    assert float((out.double() - want).abs().max()) <= 2e-5 * scale


@pytest.mark.parametrize("storage,metric,d,nq,nb,k", [
    (0, O.METRIC_L2, 96, 300, 140_001, 100), (0, O.METRIC_INNER_PRODUCT, 192, 129, 131_328, 10),
    (0, O.METRIC_L2, 128, 1000, 70_000, 5), (1, O.METRIC_L2, 40, 513, 131_329, 1024),
    (2, O.METRIC_INNER_PRODUCT, 384, 257, 100_100, 32), (2, O.METRIC_L2, 64, 16_000, 33_000, 3),
    (0, O.METRIC_L2, 64, 6000, 40_000, 20)])
def test_filter(fm, res, storage, metric, d, nq, nb, k):
    xb = H.gaussian(nb, d, 1)
    xq = H.gaussian(nq, d, 2)
    idx = fm.B200IndexFlat(res, d, metric, storage)
    idx.add(xb)
    D, I = idx.search(xq, k)
    D2, I2 = idx.search(xq, k)   # candidates come in any order, results do not
    assert np.array_equal(D, D2) and np.array_equal(I, I2)
    for q in (slice(0, 8), slice(nq // 2, nq // 2 + 8), slice(nq - 8, nq)):
        H.check_against_oracle(metric, storage, True, xb, xq[q], k, D[q], I[q], loose=False)
    idx.close()


def search_words(fm, xb, xq, storage, metric, k):
    """Result and status words of a search whose fp32 rows are two fp16 planes, which is what the resident kernel takes."""
    nb, d = xb.shape
    st = Stored(fm, xb, storage)
    xq_dev = torch.from_numpy(xq).cuda()
    D = torch.empty((len(xq), k), dtype=torch.float32, device="cuda:0")
    I = torch.empty((len(xq), k), dtype=torch.int64, device="cuda:0")
    a = st.args(fm, xq_dev, metric, k, 2, D, I)
    if storage == 0:
        fm.abi.check_op(fm.lib().b200f_store_rows_fp32(vp(st.rows), st.pitch, nb, d, vp(st.rows), st.pitch, vp(st.planes),
                                                       st.ppitch, nb * st.ppitch, 1, 4, None, None, 1, cur_stream()), "planes")
        a.plane_format, a.plane_scale_log2 = 1, 4
    fm.abi.check_op(fm.lib().b200f_search(ctypes.byref(a)), "search")
    torch.cuda.synchronize()
    return D.cpu().numpy(), I.cpu().numpy(), st.status.tolist()


@pytest.mark.parametrize("storage,metric,d,nq,nb,k", [
    (0, O.METRIC_L2, 96, 300, 140_001, 100), (0, O.METRIC_INNER_PRODUCT, 192, 129, 131_328, 10), (0, O.METRIC_L2, 128, 1000, 70_000, 5),
    (0, O.METRIC_L2, 184, 200, 140_001, 1024), (1, O.METRIC_L2, 40, 513, 131_329, 1024), (2, O.METRIC_INNER_PRODUCT, 384, 257, 100_100, 32)])
def test_no_hit_is_lost(fm, res, storage, metric, d, nq, nb, k):
    # rows that lost hits, or took too many, would be redone and come out right all the same: none is
    xb = H.gaussian(nb, d, 1)
    xq = H.gaussian(nq, d, 2)
    D, I, words = search_words(fm, xb, xq, storage, metric, k)
    assert words[:2] == [0, 0]
    for q in (slice(0, 8), slice(nq - 8, nq)):
        H.check_against_oracle(metric, storage, True, xb, xq[q], k, D[q], I[q], loose=False)


@pytest.mark.parametrize("storage", [0, 1, 2])
@pytest.mark.parametrize("near,first", [(3, 0), (32, 0), (32, 17), (100, 5)])
@pytest.mark.parametrize("nq", [129, 300])
def test_hits_of_all_rows_in_one_chunk(fm, res, storage, near, first, nq):
    # queries near one another and a block of rows near them, in a tile that no sample takes: every row of a warp hits every
    # column of a chunk of 32, four turns of eight rows, and the queue is worked off in the middle of it.  What the
    # threshold admits beside them still fits the buffers, so nothing is redone.  (Around the origin: elsewhere their
    # distances would be small differences of large products.)
    nb, d, k = 140_000, 64, 20
    xb = H.gaussian(nb, d, 3)
    at = 512 * 133 + first
    xb[at:at + near] = H.gaussian(near, d, 5, scale=0.2)
    xq = H.gaussian(nq, d, 6, scale=0.2)
    D, I, words = search_words(fm, xb, xq, storage, O.METRIC_L2, k)
    assert words[:2] == [0, 0]
    m = min(near, k)
    assert ((I[:, :m] >= at) & (I[:, :m] < at + near)).all()
    for q in (slice(0, 4), slice(nq - 4, nq)):
        H.check_against_oracle(O.METRIC_L2, storage, True, xb, xq[q], k, D[q], I[q], loose=False)


@pytest.mark.parametrize("storage,nq,k", [(2, 129, 10), (1, 300, 100), (0, 257, 10), (2, 300, 1000)])
def test_overflowed_rows_stop_filtering(fm, res, storage, nq, k):
    # equal rows: every column is a hit of every query.  What a search over them pays for a filter that is in vain stays
    # within what the redo without one takes; hits that no longer fit used to be worked off one by one (5 times as long)
    nb, d = 1_000_000, 24
    idx = fm.B200IndexFlat(res, d, O.METRIC_L2, storage)
    idx.add(np.tile(H.gaussian(1, d, 1), (nb, 1)))
    xq = torch.from_numpy(H.gaussian(nq, d, 2)).cuda()
    best = {}
    try:
        for mode in (0, 2):   # auto, without the filter
            assert fm.lib().b200f_set_selection_mode(mode) == 0
            t = []
            for _ in range(5):
                t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                t0.record()
                D, I = idx.search(xq, k)
                t1.record()
                torch.cuda.synchronize()
                assert (I == torch.arange(k, device=I.device)).all()
                t.append(t0.elapsed_time(t1))
            best[mode] = min(t)
    finally:
        fm.lib().b200f_set_selection_mode(0)
    assert best[0] <= 2 * best[2] + 0.2, best
    idx.close()


@pytest.mark.parametrize("storage,d", [(1, 256), (0, 96)])
def test_redos_of_few_rows_use_the_whole_gpu(fm, res, storage, d):
    # 100 rows are one query block, whatever the number of queries: redoing them must not take longer because the others
    # are more (ranges made for eight blocks left one to nine of 72 CTA pairs: 1,370 us instead of 590)
    nb, k = 1_000_000, 100
    xb = H.gaussian(nb, d, 1)
    xb[5000:20000] = xb[7]
    idx = fm.B200IndexFlat(res, d, O.METRIC_L2, storage)
    idx.add(xb)
    extra = []
    for nq in (1000, 2048):
        best = []
        for redone in (0, 100):
            xq = H.gaussian(nq, d, 2)
            xq[:redone] = xb[7] + H.gaussian(redone, d, 3, scale=0.01)
            xq = torch.from_numpy(xq).cuda()
            t = []
            for _ in range(8):
                t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                t0.record()
                D, I = idx.search(xq, k)
                t1.record()
                torch.cuda.synchronize()
                t.append(1e3 * t0.elapsed_time(t1))
            best.append(min(t))
        assert (I[:100] == I[0]).all() and int(I[0, 0]) == 7 and int(I[0, 1]) == 5000
        extra.append(best[1] - best[0])
    assert extra[1] <= 1.4 * extra[0], extra
    idx.close()


def test_hits_side_by_side_are_shared_out(fm, res):
    # 15,000 equal rows in a row: the hits of 100 queries near them lie in 59 neighbouring tiles.  Dealt out as ranges of
    # neighbours these were the work of three CTA pairs of 72; scattered over the index the same rows are the measure
    nb, d, nq, k = 100_000, 128, 1000, 1000
    near = np.arange(5000, 20000)
    scattered = np.sort(np.random.default_rng(1).permutation(nb)[:15000])
    best = []
    for where in (scattered, near):
        xb = H.gaussian(nb, d, 1)
        xb[where] = H.gaussian(1, d, 2)
        idx = fm.B200IndexFlat(res, d, O.METRIC_L2, 0)
        idx.add(xb)
        xq = H.gaussian(nq, d, 3)
        xq[:100] = xb[where[0]] + H.gaussian(100, d, 4, scale=0.01)
        xq = torch.from_numpy(xq).cuda()
        t = []
        for _ in range(8):
            t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            t0.record()
            D, I = idx.search(xq, k)
            t1.record()
            torch.cuda.synchronize()
            t.append(1e3 * t0.elapsed_time(t1))
        best.append(min(t))
        assert (I[:100].cpu().numpy() == where[:k]).all()
        idx.close()
    assert best[1] <= 1.15 * best[0], best
