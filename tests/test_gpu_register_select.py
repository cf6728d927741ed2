"""Selection from rows that fit a CTA's registers, counted into buckets of equal width: row lengths around ten words per
thread, results of a few up to all of them, keys that spread, tie, hold one far nearer than the rest or none at all."""
import numpy as np
import pytest

import helpers as H
from oracle import flat_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["spread", "ties", "itself", "same"])
@pytest.mark.parametrize("nb", [9, 64, 1279, 1281, 2560, 5121, 10_239, 10_241])
@pytest.mark.parametrize("k", [3, 33, 400, 2000])
def test_key_matrix(fm, res, kind, nb, k):
    # nine queries and more on up to 32,768 rows: the keys of all rows, one CTA a query
    d, nq = 16, 12
    xb = H.gaussian(nb, d, 1)
    xq = H.gaussian(nq, d, 2)
    if kind == "ties":
        xb = np.round(xb)
        xb[:, 2:] = 0
    if kind == "same":
        xb[:] = xb[0]
    if kind == "itself":
        xb += 50.0          # all rows about equally far, but for the query itself
        xq[:] = 0
        xb[nb // 2] = 0
    idx = fm.B200IndexFlat(res, d, O.METRIC_L2, 0)
    idx.set_path(2)
    idx.add(xb)
    D, I = idx.search(xq, k)
    # keys of rows around 50 carry 2^-22 (||q|| + ||x||)^2: 1e-6 of the distance
    H.check_against_oracle(O.METRIC_L2, 0, True, xb, xq, k, D, I, loose=False)
    live = min(k, nb)
    for q in range(nq):
        assert len(set(I[q, :live].tolist())) == live and (I[q, live:] == -1).all()
    if kind == "same":
        assert (I[:, :live] == np.arange(live)).all()
    idx.close()


@pytest.mark.parametrize("storage,metric", [(0, O.METRIC_L2), (1, O.METRIC_INNER_PRODUCT)])
@pytest.mark.parametrize("nq,k", [(1, 10), (4, 200), (200, 10), (200, 1024)])
def test_lists_and_candidates(fm, res, storage, metric, nq, k):
    # lists with empty places (scan, k <= 32), candidates of scans and of the tensor path
    nb, d = 70_000, 32
    xb = H.gaussian(nb, d, 3)
    xb[1000:1040] = xb[1000]
    xq = H.gaussian(nq, d, 4)
    xq[0] = xb[1000]
    idx = fm.B200IndexFlat(res, d, metric, storage)
    idx.add(xb)
    D, I = idx.search(xq, k)
    # the streaming scan of 16-bit rows rounds the queries as the tensor path does
    H.check_against_oracle(metric, storage, nq > 8 or (storage == 1 and k <= 32), xb, xq[:20], k, D[:20], I[:20], loose=False)
    idx.close()
