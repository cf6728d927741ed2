"""Thresholds from the smallest keys of 32 columns each: ragged last tiles, fewer groups than a row has threads, samples
that keep all keys, ranks from a few to hundreds.  Such a threshold admits the k best and not many more: no row is redone."""
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
