"""IVFPQ search of wide codes with a bound on the k-th distance (k > 48): every code width, both
encodings, sub-vectors of 1 to 8, lists of a few vectors, ties beyond the sort, k beyond what is visited."""
import numpy as np
import pytest

from indexsdk_b200 import datasets
from test_ivfpq_short_gpu import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("resid", [False, True])
@pytest.mark.parametrize("M,d,nlist,n,nq,nprobe,k", [
    (16, 128, 8, 20000, 3, 8, 49),
    (16, 64, 300, 9000, 700, 100, 64),       # lists of about thirty vectors
    (32, 32, 16, 30000, 40, 16, 300),        # sub-vectors of one
    (48, 96, 64, 40000, 300, 32, 100),
    (64, 128, 8, 6000, 1, 8, 1024),
    (64, 64, 4, 2200, 5, 4, 1024),
    (16, 48, 1100, 12000, 9, 1024, 50),      # the largest number of staged probes
])
def test_wide_codes_large_k(b200, resid, M, d, nlist, n, nq, nprobe, k):
    xb, _ = datasets.mixture(n, d, max(nlist // 3, 4), seed=4)
    xq, _ = datasets.mixture(nq, d, max(nlist // 3, 4), seed=5, centers_seed=4)
    ids = np.random.default_rng(1).permutation(n).astype(np.int64) * 3 - 1000
    cent, cb = datasets.train_ivfpq(xb[:6000], min(nlist, 300), M, resid, niter=2)
    if nlist > 300:
        cent = np.concatenate([cent + np.float32(0.01 * i) for i in range(4)])[:nlist]
    ix = _check(b200, xb, ids, cent, cb, resid, xq, nprobe, k)
    assert ix.stats()["fallback_queries"] == 0


@pytest.mark.parametrize("resid", [False, True])
@pytest.mark.parametrize("copies", [3000, 40000])
def test_equal_codes(b200, resid, copies):
    d, M, nlist, k = 64, 16, 4, 60
    xb, _ = datasets.mixture(2000, d, 4, seed=4)
    cent, cb = datasets.train_ivfpq(xb, nlist, M, resid, niter=2)
    xb = np.concatenate([xb, np.repeat(xb[:1], copies, axis=0)])
    ids = np.random.default_rng(2).permutation(len(xb)).astype(np.int64) - 500
    ix = _check(b200, xb, ids, cent, cb, resid, xb[:3], 4, k)
    assert (ix.stats()["fallback_queries"] > 0) == (copies == 40000)   # more than a candidate row holds
