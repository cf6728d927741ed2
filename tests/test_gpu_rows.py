"""store_rows / load_rows at the row lengths where their vector width, lanes per row and pads change,
and the storage an index keeps between reset() and the next add()."""
import ctypes

import numpy as np
import pytest

import helpers as H
from oracle import flat_oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("storage", [0, 1, 2])
@pytest.mark.parametrize("d", [1, 2, 4, 6, 7, 8, 12, 31, 32, 36, 66, 100, 127, 132, 520, 770, 1028])
def test_store_and_load_rows(fm, res, storage, d):
    from test_gpu_ops import Stored, cur_stream, vp
    n = 61 if d > 64 else 1003   # not a multiple of the rows a warp takes
    xb = H.uniform_pm1(n, d, d)
    st = Stored(fm, xb, storage)
    eff = O.round_storage(xb, storage)
    # squares of d values <= 1 summed in fp32 in any order: d * 2^-24 relative, below 1e-4 for d <= 1028
    np.testing.assert_allclose(st.norms[:n].cpu().numpy(), O.row_norms(eff), rtol=(d + 4) * 2.0 ** -24)
    back = torch.full((n, d), float("nan"), device="cuda:0")
    fm.abi.check_op(fm.lib().b200f_load_rows(vp(st.rows), storage, n, d, st.pitch, vp(back), cur_stream()), "load_rows")
    assert np.array_equal(back.cpu().numpy().view(np.uint32), eff.view(np.uint32))
    if storage == 0:
        assert not st.rows.view(torch.float32).reshape(n, st.pitch)[:, d:].any()       # pads are zero
        planes = st.planes.view(torch.bfloat16).reshape(3, n, st.ppitch).to(torch.float64)
        np.testing.assert_allclose(planes[:, :, :d].sum(0).cpu().numpy(), xb.astype(np.float64), rtol=2.0 ** -22, atol=1e-30)
        assert not planes[:, :, d:st.ppitch - 8].any() and not planes[1:, :, d:].any()
    else:
        bits = st.rows.view(torch.int16).reshape(n, st.pitch)
        assert not bits[:, d:st.pitch - 8].any() and not bits[:, st.pitch - 4:].any()


@pytest.mark.parametrize("storage", [0, 1])
def test_storage_kept_by_reset(fm, res, storage):
    # refilled with fewer, more and equally many rows, beside a second index that resets in between
    d = 72
    xb = H.uniform_pm1(9000, d, 3)
    xq = H.uniform_pm1(12, d, 4)
    a = fm.B200IndexFlat(res, d, O.METRIC_L2, storage)
    b = fm.B200IndexFlat(res, d, O.METRIC_INNER_PRODUCT, storage)
    for n in (5000, 1200, 9000, 9000):
        a.add(xb[:n])
        b.add(xb[:n // 2])
        b.reset()
        assert b.ntotal == 0 and b.device_rows() == 0
        assert np.array_equal(a.reconstruct_n(0, n), O.round_storage(xb[:n], storage))
        D, I = a.search(xq, 10)
        H.check_against_oracle(O.METRIC_L2, storage, True, xb[:n], xq, 10, D, I)
        a.reset()
        assert a.ntotal == 0 and a.device_rows() == 0
    a.set_growth_mode(1)           # retained storage is dropped when the index changes its growth mode
    a.add(xb)
    assert np.array_equal(a.reconstruct_n(0, 9000), O.round_storage(xb, storage))
    a.close()
    b.close()


def test_reset_gives_back_what_exceeds_the_bound(fm, res):
    # 9.2 GB of rows: more than an index may keep, so reset() returns the memory to the device
    d = 768
    n = 3_000_000
    x = torch.zeros((250_000, d), device="cuda:0")
    idx = fm.B200IndexFlat(res, d, O.METRIC_INNER_PRODUCT, 0)
    free0 = torch.cuda.mem_get_info()[0]
    idx.reserve(n)
    idx.add(x)
    assert free0 - torch.cuda.mem_get_info()[0] > 8 << 30
    idx.reset()
    assert free0 - torch.cuda.mem_get_info()[0] < 1 << 30
    idx.close()


def test_what_reset_keeps_is_given_back(fm, res):
    # 4.3 GB of an empty index, on request
    idx = fm.B200IndexFlat(res, 768, O.METRIC_INNER_PRODUCT, 1)
    res.release_retained()
    torch.cuda.empty_cache()
    free0 = torch.cuda.mem_get_info()[0]
    xb = H.uniform_pm1(500, 768, 5)

    def used():
        return free0 - torch.cuda.mem_get_info()[0]

    for _ in range(2):
        idx.reserve(2_800_000)
        idx.add(xb)
        assert used() > 4 << 30
        idx.reset()
        assert used() > 4 << 30
        assert res.release_retained() > 4 << 30
        assert used() < 1 << 28 and res.release_retained() == 0
    idx.add(xb)
    assert np.array_equal(idx.reconstruct_n(0, 500), O.round_storage(xb, 1))
    idx.close()


@pytest.mark.parametrize("n", [8192, 30_000])
def test_plane_scale_from_a_sample(fm, res, n):
    # one row 600 times larger than the others: over fp16's range at a scale made for them (2^7), while they
    # stay inside it (0.95 / 8 >= 2^-4) at the scale made for it; of 30,000 rows the sample takes every third
    d = 48
    xb = H.uniform_pm1(n, d, 11)
    xb[n - 2] *= np.float32(600.0)
    idx = fm.B200IndexFlat(res, d, O.METRIC_L2, 0)
    idx.add(xb)
    assert idx.fp32_planes == fm.abi.PLANES_FP16X2
    xq = H.uniform_pm1(40, d, 12)
    D, I = idx.search(xq, 10)
    H.check_against_oracle(O.METRIC_L2, 0, True, xb, xq, 10, D, I)
    idx.close()


@pytest.mark.parametrize("row", [2, 20_000])
def test_a_row_far_shorter_than_the_others(fm, res, row):
    # below 2^-4 at any scale that fits the others (sampled or not): three bf16 planes
    n, d = 30_000, 48
    xb = H.uniform_pm1(n, d, 13)
    xb[row] *= np.float32(2.0 ** -12)
    xb[row + 2] *= np.float32(600.0)
    idx = fm.B200IndexFlat(res, d, O.METRIC_INNER_PRODUCT, 0)
    idx.add(xb)
    assert idx.fp32_planes == fm.abi.PLANES_BF16X3
    xq = H.uniform_pm1(40, d, 12)
    D, I = idx.search(xq, 10)
    H.check_against_oracle(O.METRIC_INNER_PRODUCT, 0, True, xb, xq, 10, D, I)
    idx.close()


@pytest.mark.parametrize("where", ["device", "host", "second_add"])
@pytest.mark.parametrize("d", [48, 128, 1536])
@pytest.mark.parametrize("factor", [20, 50, 100, 250])
def test_a_row_far_longer_than_the_sample(fm, res, where, d, factor):
    # one row the sample does not take (it takes every third), its elements inside fp16's range at a scale made for
    # the others but its norm beyond what the norm columns hold: found on the tensor path all the same
    n, nq, k, row = 30_000, 12, 5, 20_000
    xb = H.uniform_pm1(n, d, 13)
    xb[row] *= np.float32(factor)
    xq = H.uniform_pm1(nq, d, 14)
    xq[3] = xb[row]
    idx = fm.B200IndexFlat(res, d, O.METRIC_L2, 0)
    if where == "host":
        idx.add(xb)
    elif where == "device":
        idx.add(torch.from_numpy(xb).to("cuda:0"))
        # at the scale made for the long row the others keep 0.9 * 64 / 250 > 2^-4
        assert idx.fp32_planes == fm.abi.PLANES_FP16X2
    else:
        idx.add(torch.from_numpy(xb[:row]).to("cuda:0"))
        idx.add(torch.from_numpy(xb[row:]).to("cuda:0"))
    D, I = idx.search(xq, k)
    assert I[3, 0] == row
    x64, q64 = xb.astype(np.float64), xq.astype(np.float64)
    length = np.sqrt((x64 ** 2).sum(1))
    for q in range(nq):
        true = ((x64 - q64[q]) ** 2).sum(1)
        want = np.sort(np.partition(true, k - 1)[:k])
        # 22-bit products: 2^-21 (||q|| + ||x||)^2 of a distance.  Their fp32 sum grows 16 columns at a time, d / 16 + 1
        # steps, each dropping up to 2^-23 of a sum of at most ||q|| ||x||, of which a distance takes twice: another
        # (d / 16 + 1) 2^-24 (||q|| + ||x||)^2, 5.8e-6 for d = 1536, where the distance of the long row to itself came
        # out as 6.5e-6 ||x||^2
        tol = (2.0 ** -21 + (d / 16 + 1) * 2.0 ** -24) * (np.sqrt((q64[q] ** 2).sum()) + length[I[q]].max()) ** 2
        assert np.abs(D[q] - want).max() <= tol and np.abs(true[I[q]] - D[q]).max() <= tol
    idx.close()
