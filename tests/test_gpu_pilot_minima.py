"""Thresholds from the smallest keys of four columns each: ragged last tiles, fewer groups than a row has threads, samples
that keep all keys, ranks from a few to hundreds.  Such a threshold admits the k best and not many more: no row is redone;
of rows stored in runs of near ones it admits more, but not so many that most queries are."""
import ctypes

import numpy as np
import pytest
import torch

import helpers as H
from oracle import flat_oracle as O
from test_gpu_ops import Stored

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,metric", [(1, O.METRIC_L2), (2, O.METRIC_INNER_PRODUCT), (0, O.METRIC_L2)])
@pytest.mark.parametrize("nq,nb,k", [(9, 33_000, 3), (50, 300_007, 2048), (129, 131_073, 100), (300, 140_033, 10),
                                     (20, 262_400, 1000), (600, 100_001, 32), (1000, 524_289, 5)])
def test_thresholds_hold(fm, res, storage, metric, nq, nb, k):
    d = 24
    xb = H.gaussian(nb, d, 1)
    xq = H.gaussian(nq, d, 2)
    st = Stored(fm, xb, storage)
    xq_dev = torch.from_numpy(xq).cuda()
    D = torch.empty((nq, k), dtype=torch.float32, device="cuda:0")
    I = torch.empty((nq, k), dtype=torch.int64, device="cuda:0")
    a = st.args(fm, xq_dev, metric, k, 2, D, I)
    fm.abi.check_op(fm.lib().b200f_search(ctypes.byref(a)), "search")
    torch.cuda.synchronize()
    assert st.status.tolist()[:2] == [0, 0]
    D, I = D.cpu().numpy(), I.cpu().numpy()
    for q in (slice(0, 4), slice(nq - 4, nq)):
        H.check_against_oracle(metric, storage, True, xb, xq[q], k, D[q], I[q], loose=False)


@pytest.mark.parametrize("storage,metric", [(2, O.METRIC_L2), (0, O.METRIC_L2), (1, O.METRIC_INNER_PRODUCT)])
@pytest.mark.parametrize("run", [8, 16, 32])
@pytest.mark.parametrize("nq,k", [(1000, 10), (1000, 100), (120, 100)])
def test_rows_in_runs_of_near_ones(fm, res, storage, metric, run, nq, k):
    # chunks of a document, augmentations of an image.  A sample of whole tiles holds a run or none of it, so some
    # queries are redone whatever the threshold: simulated with minima over four neighbouring columns (the
    # threads' loads of four keys) 1 to 32 % of them, over 32 columns 39 to 100 %; the bound leaves three deviations of a
    # count with that share
    nb, d = 1_000_000, 24
    xb = np.repeat(H.gaussian(nb // run, d, 11), run, axis=0) + H.gaussian(nb, d, 12, scale=0.05)
    if metric == O.METRIC_INNER_PRODUCT:
        xb /= np.linalg.norm(xb, axis=1, keepdims=True)
    xq = H.gaussian(nq, d, 13)
    st = Stored(fm, xb, storage)
    xq_dev = torch.from_numpy(xq).cuda()
    D = torch.empty((nq, k), dtype=torch.float32, device="cuda:0")
    I = torch.empty((nq, k), dtype=torch.int64, device="cuda:0")
    a = st.args(fm, xq_dev, metric, k, 2, D, I)
    fm.abi.check_op(fm.lib().b200f_search(ctypes.byref(a)), "search")
    torch.cuda.synchronize()
    status = st.status.tolist()
    assert status[0] == 0 and status[1] <= 0.32 * nq + 1.5 * nq ** 0.5, status
    H.check_against_oracle(metric, storage, True, xb, xq[:2], k, D[:2].cpu().numpy(), I[:2].cpu().numpy(), loose=False)
