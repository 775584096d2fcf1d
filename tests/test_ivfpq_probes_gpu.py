"""IVFPQ search whose probe selection outgrows its candidate lists: thousands of centroids closer together
than the coarse filter can tell apart.  Such queries are searched again behind the others of their batch."""
import numpy as np
import pytest

import oracle
from helpers import assert_exact
from indexsdk_b200 import datasets

pytestmark = pytest.mark.gpu
L2 = 1


# copies: survivors of the fused tail's pruning beyond what it holds (1 100), candidates beyond the row (2 500);
# nprobe above and below what the fused tail takes
@pytest.mark.parametrize("resid", [False, True])
@pytest.mark.parametrize("M,k,nq,exact", [(8, 70, 40, False),       # scan with a bound, short codes
                                          (16, 60, 40, False),      # ... wide codes
                                          (16, 10, 40, False),      # filter, one block per query and split
                                          (16, 10, 1300, False),    # filter, persistent blocks
                                          (4, 10, 40, True)])       # exact scan
@pytest.mark.parametrize("nlist,copies,nprobe", [(3000, 1100, 96), (3000, 2500, 96), (9700, 9000, 300)])
def test_probes_that_outgrow_their_lists(b200, monkeypatch, resid, M, k, nq, exact, nlist, copies, nprobe):
    d, n = 16, 20000
    if nq > 100 and nlist > 3000:
        pytest.skip("the same code as with fewer lists")
    rng = np.random.default_rng(1)
    monkeypatch.setenv("B200IDX_IVFPQ_EXACT", "1" if exact else "0")
    cent = datasets.gaussian(nlist, d, seed=1)
    cent[:copies] = cent[:1] + np.float32(1e-4) * datasets.gaussian(copies, d, seed=2)
    cb = np.float32(0.1) * rng.standard_normal((M, 256, d // M)).astype(np.float32)
    ix = b200.IndexIVFPQ(d, nlist, M, 8, by_residual=resid)
    ix.set_centroids(cent)
    ix.set_codebooks(cb)
    ln = rng.integers(0, nlist, size=n).astype(np.int32)
    codes = rng.integers(0, 256, size=(n, M), dtype=np.uint8)
    ids = rng.permutation(n).astype(np.int64)
    ix.add_codes(ln, codes, ids)
    ix.nprobe = nprobe
    xq = datasets.gaussian(nq, d, seed=3)
    xq[::3] = cent[:1] + np.float32(0.05) * xq[::3]        # these queries' probes are among the copies
    D, I = ix.search(xq, k)
    off, cs, idl = oracle.build_lists(ln, codes, ids, nlist)
    Dr, Ir = oracle.ivfpq_search(cent, cb, resid, off, cs, idl, xq, nprobe, k)
    assert_exact(D, I, Dr, Ir)
    if not exact:   # every probed list is visited once (the exact scan does not count)
        probes = oracle.flat_search(L2, cent, xq, nprobe)[1]
        assert ix.stats()["scan_codes"] == int((off[1:] - off[:-1])[probes].sum())
