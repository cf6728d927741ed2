"""row_select: the result lists of the streaming scans and of the fused kernel, and filtered candidates, at
the list lengths, row counts and ties where the selection changes its way (bound from thread minima or
exact radix select, placing by counting or by sorted runs), against the oracle and the sorting kernel."""
import numpy as np
import pytest

import helpers as H
from oracle import flat_oracle as O

pytestmark = pytest.mark.gpu


def tied(nb, d, seed):
    """Rows of which a few hundred are exact copies of one row, spread over the shard."""
    xb = H.gaussian(nb, d, seed)
    xb[200:500] = xb[17]
    xb[nb // 3::max(1, nb // 211)] = xb[17]
    return xb


@pytest.mark.parametrize("storage", [0, 1])
@pytest.mark.parametrize("nb", [1, 31, 3000, 150_000])
@pytest.mark.parametrize("nq,k", [(1, 1), (1, 32), (3, 10), (8, 31), (40, 1), (40, 32)])
def test_partial_lists(fm, res, storage, nb, nq, k):
    # scan lists (nq <= 8) and the fused kernel's lists; k above nb leaves empty slots
    xb = tied(nb, 24, nb) if nb > 500 else H.gaussian(nb, 24, nb)
    xq = H.gaussian(nq, 24, 1000 + nq)
    if nb > 500:
        xq[0] = xb[17] + 0.3           # the copies fill its list: ties go to the lower label
    L = fm.lib()
    assert L.b200f_set_selection_mode(2) == 0
    try:
        idx = fm.B200IndexFlat(res, 24, O.METRIC_L2, storage)
        idx.add(xb)
        D, I = idx.search(xq, k)
    finally:
        L.b200f_set_selection_mode(0)
    tensor = nq > 8 or (storage == 1 and nb > 100_000)   # the streaming kernel rounds the query like the tensor path
    H.check_against_oracle(O.METRIC_L2, storage, tensor, xb, xq, k, D, I, loose=False)
    if nb > 500:
        assert I[0, 0] == 17 and list(I[0]) == sorted(I[0])
    if k > nb:
        assert (I[:, nb:] == -1).all() and np.isposinf(D[:, nb:]).all()
    idx.close()


@pytest.mark.parametrize("nq", [20, 700])
@pytest.mark.parametrize("k", [1, 2, 32, 64, 65, 128, 129, 1024])
def test_filtered_candidates_match_sorting_kernel(fm, res, nq, k):
    nb, d = 140_000, 32
    xb = tied(nb, d, 7)
    xq = H.gaussian(nq, d, 8)
    xq[::7] = xb[17] + 0.02
    L = fm.lib()
    idx = fm.B200IndexFlat(res, d, O.METRIC_L2, 1)
    idx.add(xb)
    idx.set_path(2)
    assert L.b200f_set_selection_mode(1) == 0
    try:
        D1, I1 = idx.search(xq, k)
        assert L.b200f_set_rank_select(0) == 0
        D0, I0 = idx.search(xq, k)
    finally:
        L.b200f_set_rank_select(1)
        L.b200f_set_selection_mode(0)
    assert np.array_equal(I1, I0) and np.array_equal(D1, D0)
    idx.close()
