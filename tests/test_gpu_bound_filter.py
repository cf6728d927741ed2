"""Streaming scans with k > 32 whose filter keys are bounds of the true ones (L2, from 32 Mi stored elements on), the
candidates scored again in fp32: on data the bounds fit and on data where the exact filter has to run."""
import numpy as np
import pytest

from oracle import flat_oracle as O

pytestmark = pytest.mark.gpu

# ||q||^2 + ||x||^2 - 2 q.x from 22-bit products: 2^-22 (||q|| + ||x||)^2 for the dropped bits, as much again for the sums
TOL = 2.0 ** -21


def check(xb, xq, k, D, I):
    xb = xb.astype(np.float64)
    for q in range(len(xq)):
        true = np.square(xb - xq[q].astype(np.float64)).sum(1)
        tol = TOL * (np.linalg.norm(xq[q]) + np.sqrt(np.square(xb).sum(1).max())) ** 2
        want = np.sort(np.partition(true, k - 1)[:k])
        assert np.abs(D[q] - want).max() <= tol
        assert np.abs(true[I[q]] - D[q]).max() <= tol
        assert len(set(I[q].tolist())) == k
        assert (np.diff(D[q]) >= 0).all()


def rows(kind, n, d, seed, where):
    """where: the centre of `near` data, the same for rows and queries."""
    x = np.random.default_rng(seed).standard_normal((n, d), dtype=np.float32)
    return x if kind == "around" else where + x * np.float32(0.03 if kind == "far" else 1e-5)


@pytest.mark.parametrize("storage", [0, 1, 2])
@pytest.mark.parametrize("kind", ["around", "far", "tiny", "huge_query"])
@pytest.mark.parametrize("nq,k", [(2, 33), (5, 200), (8, 1025)])
def test_scans(fm, res, storage, kind, nq, k):
    nb, d = 700_001, 48
    where = np.full(d, 0.0 if kind == "tiny" else 1.5, np.float32)
    data = kind if kind in ("far", "tiny") else "around"
    xb = rows(data, nb, d, 3, where)
    xq = rows(data, nq, d, 4, where)
    if kind == "huge_query":
        xq[1, :3] = (70_000, -40_000, 3)
    idx = fm.B200IndexFlat(res, d, O.METRIC_L2, storage)
    idx.add(xb)
    D, I = idx.search(xq, k)
    check(O.round_storage(xb, storage), xq, k, D, I)
    idx.close()
