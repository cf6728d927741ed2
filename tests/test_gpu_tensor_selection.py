"""Selection on the tensor path at the sizes where its stages change: the whole key matrix (up to 32,768 rows
and 16 Mi pairs), thresholds from samples of different density, and k beyond 1024."""
import numpy as np
import pytest

import helpers as H
from oracle import flat_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,metric", [(0, O.METRIC_L2), (1, O.METRIC_INNER_PRODUCT), (2, O.METRIC_L2)])
@pytest.mark.parametrize("nq,nb,k", [(9, 1, 3), (130, 255, 300), (17, 32_768, 10), (17, 32_769, 10), (512, 32_768, 33),
                                     (40, 32_768, 1500), (11, 32_769, 1025), (300, 60_000, 4096), (129, 140_001, 100)])
def test_stages(fm, res, storage, metric, nq, nb, k):
    d = 40
    xb = H.gaussian(nb, d, 1)
    xq = H.gaussian(nq, d, 2)
    idx = fm.B200IndexFlat(res, d, metric, storage)
    idx.add(xb)
    D, I = idx.search(xq, k)
    H.check_against_oracle(metric, storage, True, xb, xq[:40], k, D[:40], I[:40], loose=False)
    H.check_against_oracle(metric, storage, True, xb, xq[-3:], k, D[-3:], I[-3:], loose=False)
    idx.close()


@pytest.mark.parametrize("storage", [0, 2])
@pytest.mark.parametrize("k", [10, 100, 2000])
def test_rows_the_sample_misjudges(fm, res, storage, k):
    # the first tiles hold every near row of query 0 (the sample sees them all, or too few of them), and query 1
    # finds one row 30,000 times, more than its candidate buffer holds
    # ||q||^2 + ||x||^2 - 2 q.x in 22 bits leaves 2^-22 (||q|| + ||x||)^2 of a distance: 9e-5 of 0.24 d / 24 for
    # query 1, 7e-5 of about 1.3 for query 0 (a cluster of sigma 0.3 around 2; of sigma 0.1 around 5 it would be 6e-3)
    nb, nq, d = 120_000, 64, 24
    xb = H.gaussian(nb, d, 3)
    xb[:512] = 2.0 + 0.3 * H.gaussian(512, d, 4)
    xb[80_000:110_000] = xb[80_000]
    xq = H.gaussian(nq, d, 5)
    xq[0] = 2.0
    xq[1] = xb[80_000] + np.float32(0.1)
    idx = fm.B200IndexFlat(res, d, O.METRIC_L2, storage)
    idx.add(xb)
    D, I = idx.search(xq, k)
    H.check_against_oracle(O.METRIC_L2, storage, True, xb, xq[:8], k, D[:8], I[:8], loose=False)
    idx.close()


@pytest.mark.parametrize("storage,metric", [(2, O.METRIC_INNER_PRODUCT), (2, O.METRIC_L2)])
@pytest.mark.parametrize("nb", [3000, 32_768, 32_769, 140_000, 600_000])
@pytest.mark.parametrize("k", [2, 10, 32, 100, 1000])
def test_infinite_keys_are_no_results(fm, res, storage, metric, nb, k):
    # products (or norms) of all rows but a few overflow fp32: as in the oracle, such rows fill no slot, whichever
    # way their number selects
    nq, d, few = 20, 16, 7
    xb = np.full((nb, d), 2.0 ** 126, np.float32)
    rows = np.linspace(0, nb - 1, few).astype(int)
    xb[rows] = H.gaussian(few, d, 3)
    xq = -1.0 - np.abs(H.gaussian(nq, d, 4))
    if metric == O.METRIC_INNER_PRODUCT:
        xq *= np.float32(1024.0)
    idx = fm.B200IndexFlat(res, d, metric, storage)
    idx.add(xb)
    D, I = idx.search(xq, k)
    live = min(k, few)
    assert (np.sort(I[:, :live], axis=1) >= 0).all() and np.isin(I[:, :live], rows).all()
    assert (I[:, live:] == -1).all()
    assert (np.isposinf(D[:, live:]) if metric == O.METRIC_L2 else np.isneginf(D[:, live:])).all()
    H.check_against_oracle(metric, storage, True, xb[rows], xq, live, D[:, :live], np.searchsorted(rows, I[:, :live]))
    idx.close()


@pytest.mark.parametrize("storage", [0, 2])
def test_rows_redone_over_several_column_chunks(fm, res, storage):
    # 300 of 9,000 queries find one row 30,000 times, more than a candidate buffer holds; their key matrix has
    # 2^30 / 4 / 9,000 columns a chunk, so five stores and selections follow one another
    nb, nq, d, k = 120_000, 9_000, 24, 100
    xb = H.gaussian(nb, d, 3)
    xb[80_000:110_000] = xb[80_000]
    xq = H.gaussian(nq, d, 5)
    xq[::30] = xb[80_000] + np.float32(0.1) * H.gaussian(len(xq[::30]), d, 6)
    idx = fm.B200IndexFlat(res, d, O.METRIC_L2, storage)
    idx.add(xb)
    for _ in range(3):
        D, I = idx.search(xq, k)
        # ||q||^2 + ||x||^2 - 2 q.x in 22 bits leaves 2^-22 (||q|| + ||x||)^2 of a distance: up to 1e-4 of the 0.24
        # between such a query and its rows, within the 2e-4 of the comparison
        pick = np.r_[0:1800:30, 8970, 1:30, nq - 3:nq]
        H.check_against_oracle(O.METRIC_L2, storage, True, xb, xq[pick], k, D[pick], I[pick], loose=False)
    idx.close()


@pytest.mark.parametrize("how", ["search", "search_async"])
@pytest.mark.parametrize("nb,tail,k", [(2000, 2000, 10), (2000, 8000, 32), (5000, 900, 3), (32_768, 14_000, 10)])
def test_last_batch_that_needs_more_scratch(fm, res, how, nb, tail, k):
    # a search takes 16,384 queries at a time; the shorter rest needs more scratch than a full batch does
    size = fm.lib().b200f_search_scratch_bytes
    d, n = 32, 16_384 + tail
    assert size(tail, nb, d, k, 0, 0) > size(16_384, nb, d, k, 0, 0)
    xb = H.gaussian(nb, d, 1)
    xq = H.gaussian(n, d, 2)
    idx = fm.B200IndexFlat(res, d, O.METRIC_L2, 0)
    idx.add(xb)
    if how == "search":
        D, I = idx.search(xq, k)
    else:
        D, I = np.empty((n, k), np.float32), np.empty((n, k), np.int64)
        idx.search_async(xq, k, D, I).wait()
    idx.close()
    for q in (slice(0, 8), slice(16_380, 16_390), slice(n - 8, n)):
        H.check_against_oracle(O.METRIC_L2, 0, True, xb, xq[q], k, D[q], I[q], loose=False)
