"""Lists of the streaming scans: a warp's first rows sorted into an empty list, the warps' lists merged pair by pair,
at row counts around a warp's 32 rows, a CTA's 256 and the grid's; keys that tie, overflow or are no numbers."""
import numpy as np
import pytest

import helpers as H
from oracle import flat_oracle as O

pytestmark = pytest.mark.gpu

GRID = 3 * 148 * 8 * 32   # rows of one block per warp: three CTAs of eight warps on 148 SMs


@pytest.mark.parametrize("storage,metric", [(0, O.METRIC_L2), (0, O.METRIC_INNER_PRODUCT), (2, O.METRIC_L2)])
@pytest.mark.parametrize("nb", [1, 31, 33, 255, 257, 5000, GRID - 1, GRID + 33])
@pytest.mark.parametrize("nq,k", [(1, 1), (1, 32), (2, 10), (3, 31), (4, 32), (8, 17)])
def test_row_counts(fm, res, storage, metric, nb, nq, k):
    d = 33
    xb = H.gaussian(nb, d, 1)
    xb[nb // 2:] = xb[: nb - nb // 2]   # every row twice: ties go to the lower label
    xq = H.gaussian(nq, d, 2)
    idx = fm.B200IndexFlat(res, d, metric, storage)
    idx.set_path(1)
    idx.add(xb)
    D, I = idx.search(xq, k)
    # 16-bit rows: larger shards take the streaming kernel, which rounds the queries too
    H.check_against_oracle(metric, storage, False, xb, xq, k, D, I, strict=storage == 0)
    idx.close()


def test_keys_that_are_no_numbers_or_infinite(fm, res):
    # rows 0 .. 9 give NaN, 10 .. 19 +INF distances: the first are never returned, the second behind all others
    nb, d, k = 40, 32, 32
    xb = H.gaussian(nb, d, 3)
    xb[:10, 0] = np.nan
    xb[10:20] = 1e30
    idx = fm.B200IndexFlat(res, d, O.METRIC_L2, 0)
    idx.set_path(1)
    idx.add(xb)
    D, I = idx.search(H.gaussian(1, d, 4), k)
    assert sorted(I[0, :20]) == list(range(20, 40)) and np.isfinite(D[0, :20]).all()
    assert I[0, 20:30].tolist() == list(range(10, 20)) and np.isposinf(D[0, 20:30]).all()
    assert (I[0, 30:] == -1).all()
    idx.close()


@pytest.mark.parametrize("storage,d,nq", [(0, 2100, 8), (0, 257, 5), (2, 1000, 8), (1, 24, 7)])
def test_sample_of_wide_and_narrow_rows(fm, res, storage, d, nq):
    # more pieces than the sample's lanes hold at a time, and more queries than share a launch
    nb, k = 40_000, 40
    xb = H.gaussian(nb, d, 5)
    xq = H.gaussian(nq, d, 6)
    idx = fm.B200IndexFlat(res, d, O.METRIC_L2, storage)
    idx.set_path(1)
    idx.add(xb)
    D, I = idx.search(xq, k)
    H.check_against_oracle(O.METRIC_L2, storage, False, xb, xq, k, D, I, strict=storage == 0)
    idx.close()
