"""Streaming scans whose thresholds come from a sample of the rows: candidate buffers (k > 32) and lists
cut at a threshold (k <= 32), at the row counts where they begin, on rows the sample misjudges and on ties."""
import ctypes

import numpy as np
import pytest

import helpers as H
from oracle import flat_oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def redone(fm, stored, xq, metric, k, path=1):
    """Queries whose result had to be found again without the sample's threshold (status word 1), and the result."""
    q = torch.from_numpy(xq).to("cuda:0")
    D = torch.empty((len(xq), k), dtype=torch.float32, device="cuda:0")
    I = torch.empty((len(xq), k), dtype=torch.int64, device="cuda:0")
    a = stored.args(fm, q, metric, k, path, D, I)
    fm.abi.check_op(fm.lib().b200f_search(ctypes.byref(a)), "search")
    torch.cuda.synchronize()
    return int(stored.status[1]), D.cpu().numpy(), I.cpu().numpy()


@pytest.mark.parametrize("storage,metric", [(0, O.METRIC_L2), (1, O.METRIC_INNER_PRODUCT), (2, O.METRIC_L2)])
@pytest.mark.parametrize("nb", [32_767, 32_768, 100_003])
@pytest.mark.parametrize("nq,k", [(1, 33), (3, 200), (4, 4096), (8, 1000)])
def test_candidates(fm, res, storage, metric, nb, nq, k):
    d = 40
    xb = H.gaussian(nb, d, 1)
    xq = H.gaussian(nq, d, 2)
    idx = fm.B200IndexFlat(res, d, metric, storage)
    idx.add(xb)
    idx.set_path(1)
    D, I = idx.search(xq, k)
    H.check_against_oracle(metric, storage, False, xb, xq, k, D, I, loose=False)
    idx.close()


@pytest.mark.parametrize("storage", [0, 2])
@pytest.mark.parametrize("nq,k", [(1, 24), (1, 100), (5, 32), (8, 100)])
def test_rows_the_sample_misjudges(fm, res, storage, nq, k):
    # rows in groups of four and of 64 that begin with near ones, and, for the second query, one row repeated
    # 40,000 times, more than its candidate buffer holds.  Both must come out exactly.
    nb, d = 600_000, 16
    xb = H.gaussian(nb, d, 3)
    xb[::4] = 6.0 + 0.1 * H.gaussian(nb // 4, d, 4)
    xb[::64] = 3.0 + 0.1 * H.gaussian(len(xb[::64]), d, 5)
    xb[1:160_001:4] = xb[1]
    xq = H.gaussian(nq, d, 6)
    xq[0] = 2.5
    if nq > 1:
        xq[1] = xb[1] + 0.2
    for use_path in (0, 1):
        idx = fm.B200IndexFlat(res, d, O.METRIC_L2, storage)
        idx.add(xb)
        idx.set_path(use_path)
        D, I = idx.search(xq, k)
        tensor = storage != 0 and k <= 32    # the streaming kernel rounds the query like the tensor path
        H.check_against_oracle(O.METRIC_L2, storage, tensor, xb, xq, k, D, I, loose=False)
        idx.close()


@pytest.mark.parametrize("nb,k", [(66_000, 2400), (100_000, 2400), (100_000, 4096), (100_000, 100)])
def test_candidate_buffers_hold_what_the_threshold_admits(fm, res, nb, k):
    # independent rows: of 24 x 8 queries none may overflow (six deviations), whatever the rank of the threshold
    from test_gpu_ops import Stored
    d = 16
    st = Stored(fm, H.gaussian(nb, d, 1), 2)
    for seed in range(24):
        assert redone(fm, st, H.gaussian(8, d, 100 + seed), O.METRIC_L2, k)[0] == 0


def sampled_rows(nb, stride, pieces):
    """The rows a scan takes its thresholds from: one in every `stride`, as in the scan kernel.  A row of `pieces` 16-byte
    pieces belongs to up to eight lanes; eight columns of the sample share an offset."""
    per_step = 32 // min(8, 1 << (pieces - 1).bit_length())
    c = np.arange(nb // stride, dtype=np.uint64)
    j = c // (8 * per_step) * per_step + c % per_step
    return (c * stride + ((j * 2654435769 & 0xffffffff) * stride >> 32)).astype(np.int64)


@pytest.mark.parametrize("storage", [0, 2])
@pytest.mark.parametrize("nq,k", [(1, 24), (1, 100), (5, 32), (8, 100)])
def test_sampled_rows_nearer_than_all_others(fm, res, storage, nq, k):
    # 600,000 rows: the sample takes one in 64.  All it takes are nearer to the first query than any other row, so
    # that its threshold admits the 7 to 11 rows of its rank and no more: redone, and exact
    from test_gpu_ops import Stored
    nb, d = 600_000, 16
    xb = 6.0 + 0.1 * H.gaussian(nb, d, 3)
    near = sampled_rows(nb, 64, d // (8 if storage else 4))
    xb[near] = 3.0 + 0.1 * H.gaussian(len(near), d, 5)
    xq = H.gaussian(nq, d, 6)
    xq[0] = 2.5
    count, D, I = redone(fm, Stored(fm, xb, storage), xq, O.METRIC_L2, k)
    assert count == nq
    tensor = storage != 0 and k <= 32    # the streaming kernel rounds the query like the tensor path
    H.check_against_oracle(O.METRIC_L2, storage, tensor, xb, xq, k, D, I, loose=False)


@pytest.mark.parametrize("storage", [0, 2])
@pytest.mark.parametrize("period,k", [(8, 200), (16, 200), (64, 32), (64, 200)])
@pytest.mark.parametrize("first", ["nearest", "farthest"])
def test_rows_that_repeat_with_a_period(fm, res, storage, period, k, first):
    # an original and its augmentations, one after the other: the sample sees all of them alike, nothing is redone
    from test_gpu_ops import Stored
    nb, d, nq = 600_000, 32, 4
    xb = np.repeat(H.gaussian(nb // period, d, 7), period, axis=0)
    noise = H.gaussian(nb, d, 8, scale=0.7)
    own = np.arange(nb) % period == 0
    noise[own if first == "nearest" else ~own] = 0
    xb += noise
    xq = H.gaussian(nq, d, 9)
    count, D, I = redone(fm, Stored(fm, xb, storage), xq, O.METRIC_L2, k)
    assert count == 0
    tensor = storage != 0 and k <= 32
    H.check_against_oracle(O.METRIC_L2, storage, tensor, xb, xq, k, D, I, loose=False)
