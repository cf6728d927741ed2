"""Query counts around 16, 32 and 64: up to 64 queries are a tile of 64 rows, sixteen in every lane quarter of the accumulator,
beyond it they fill 128.  Every mode of the distance GEMM: matrix (whole sectors and ragged), lists, thresholds and their candidates."""
import ctypes

import numpy as np
import pytest
import torch

import helpers as H
from oracle import flat_oracle as O
from test_gpu_ops import Stored, cur_stream, vp

pytestmark = pytest.mark.gpu

COUNTS = (1, 8, 15, 16, 17, 31, 32, 33, 48, 49, 63, 64, 65)


@pytest.mark.parametrize("nq", COUNTS)
@pytest.mark.parametrize("storage,metric,nb", [(1, O.METRIC_L2, 4096), (2, O.METRIC_INNER_PRODUCT, 4099), (0, O.METRIC_L2, 777)])
def test_matrix(fm, res, storage, metric, nq, nb):
    d = 72
    xb = H.uniform_pm1(nb, d, 99)
    xq = H.uniform_pm1(nq, d, 77)
    st = Stored(fm, xb, storage)
    xq_dev = torch.from_numpy(xq).cuda()
    out = torch.full((nq + 1, nb), 7.0, dtype=torch.float32, device="cuda:0")
    a = st.args(fm, xq_dev, metric, 1, 2)
    fm.abi.check_op(fm.lib().b200f_pairwise(ctypes.byref(a), vp(out), nb), "pairwise")
    torch.cuda.synchronize()
    assert int(st.status[0]) == 0
    assert bool((out[nq] == 7.0).all())   # nothing behind the last query
    xb_eff, xq_eff = H.effective_operands(storage, True, xb, xq)
    want = xq_eff.astype(np.float64) @ xb_eff.astype(np.float64).T
    if metric == O.METRIC_L2:   # the squared norm of a query is that of its fp32 values
        want = (xq.astype(np.float64) ** 2).sum(1)[:, None] + (xb_eff.astype(np.float64) ** 2).sum(1)[None] - 2 * want
    # fp32 sums of at most 72 products; fp32 rows leave out 2^-24 of each
    assert np.abs(out[:nq].cpu().numpy().astype(np.float64) - want).max() <= 2e-5 * np.abs(want).max()


@pytest.mark.parametrize("nq", [c for c in COUNTS if c > 8])
@pytest.mark.parametrize("storage,metric,nb,k", [(1, O.METRIC_L2, 30_000, 1), (0, O.METRIC_INNER_PRODUCT, 20_001, 7), (2, O.METRIC_L2, 70_001, 100),
                                                 (0, O.METRIC_L2, 100_003, 10), (1, O.METRIC_INNER_PRODUCT, 150_001, 1500)])
def test_search(fm, res, storage, metric, nq, nb, k):
    d = 40
    xb = H.gaussian(nb, d, 1)
    xq = H.gaussian(nq, d, 2)
    idx = fm.B200IndexFlat(res, d, metric, storage)
    idx.add(xb)
    D, I = idx.search(xq, k)
    idx.close()
    for q in (slice(0, 2), slice(max(0, nq // 2 - 1), nq // 2 + 1), slice(nq - 2, nq)):
        H.check_against_oracle(metric, storage, True, xb, xq[q], k, D[q], I[q], loose=False)
