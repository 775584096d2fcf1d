"""PQ encoding on the device, per sub-vector length and around the tile edges, against the oracle."""
import numpy as np
import pytest

import oracle
from indexsdk_b200 import datasets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("resid", [False, True])
@pytest.mark.parametrize("d,M", [(64, 32), (64, 16), (128, 16), (64, 4), (128, 4), (48, 2), (96, 8)])
@pytest.mark.parametrize("n", [1, 255, 257, 3001])
def test_codes_vs_oracle(b200, resid, d, M, n):
    """dsub = 2, 4, 8, 16, 32 (tiled kernel) and 24, 12 (general one); exact, ties to the lower code."""
    nlist = 5
    rng = np.random.default_rng(d * M + n)
    cent = rng.standard_normal((nlist, d), dtype=np.float32)
    cb = 0.5 * rng.standard_normal((M, 256, d // M), dtype=np.float32)
    cb[:, 130] = cb[:, 7]                      # equal codewords: the first one wins
    x = datasets.gaussian(n, d, seed=n)
    x[0, :d // M] = cb[0, 7] if not resid else x[0, :d // M]
    ix = b200.IndexIVFPQ(d, nlist, M, 8, by_residual=resid)
    ix.set_centroids(cent)
    ix.set_codebooks(cb)
    ix.add(x)
    ln = oracle.ivf_assign(cent, x)
    codes = oracle.pq_encode(cb, x, resid, cent, ln)
    off, cs, ids = oracle.build_lists(ln, codes, np.arange(n, dtype=np.int64), nlist)
    for l in range(nlist):
        c, i = ix.get_list(l)
        np.testing.assert_array_equal(i, ids[off[l]:off[l + 1]])
        np.testing.assert_array_equal(c, cs[off[l]:off[l + 1]])
