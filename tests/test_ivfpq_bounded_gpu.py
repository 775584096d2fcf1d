"""IVFPQ search of wide codes with a bound on the k-th distance (k > 48): every code width, both
encodings, sub-vectors of 1 to 8, lists of a few vectors, ties beyond the sort, k beyond what is visited."""
import numpy as np
import pytest

import oracle
from helpers import assert_exact
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


def _random_codes(b200, d, M, nlist, n, resid=False):
    rng = np.random.default_rng(7)
    cent = datasets.gaussian(nlist, d, seed=1)
    cb = rng.standard_normal((M, 256, d // M)).astype(np.float32)
    ix = b200.IndexIVFPQ(d, nlist, M, 8, by_residual=resid)
    ix.set_centroids(cent)
    ix.set_codebooks(cb)
    ln = rng.integers(0, nlist, size=n).astype(np.int32)
    codes = rng.integers(0, 256, size=(n, M), dtype=np.uint8)
    ids = rng.permutation(n).astype(np.int64)
    ix.add_codes(ln, codes, ids)
    ix.nprobe = nlist
    return ix, cent, cb, oracle.build_lists(ln, codes, ids, nlist)


# lists no better than one another: about k visited / n1 vectors lie under a bound taken from n1 of them; the last
# two are more than the longest row holds, and the filter answers, not the exact scan
@pytest.mark.parametrize("M,n,k", [(16, 30000, 300), (32, 200000, 500), (16, 600000, 1000), (64, 600000, 900)])
def test_lists_without_structure(b200, M, n, k):
    ix, cent, cb, (off, cs, ids) = _random_codes(b200, M, M, 8, n)
    xq = datasets.gaussian(3, M, seed=3)
    D, I = ix.search(xq, k)
    Dr, Ir = oracle.ivfpq_search(cent, cb, False, off, cs, ids, xq, 8, k)
    assert_exact(D, I, Dr, Ir)
    assert ix.stats()["fallback_queries"] == 0


def test_scratch_follows_the_candidates_not_the_lists(b200):
    """The first large batch on an index asks for what its candidates need, not for its longest lists."""
    import torch
    ix, *_ = _random_codes(b200, 96, 48, 64, 100000)
    xq = datasets.gaussian(1000, 96, seed=3)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    ix.search(xq, 100)
    assert free - torch.cuda.mem_get_info()[0] < 200 << 20
