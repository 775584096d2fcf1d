"""Lists on their way out of an IVFPQ index (get_list): stretches of about 4 MB, both code layouts, and
merges that reuse their work arrays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,d", [(16, 16), (64, 64), (12, 48), (3, 48), (4, 16)])
@pytest.mark.parametrize("sizes", [(1, 0, 31, 33), (400000, 5, 0, 64)])
def test_lists_come_back_as_they_went_in(b200, M, d, sizes):
    rng = np.random.default_rng(M)
    ix = b200.IndexIVFPQ(d, len(sizes), M, 8, by_residual=False)
    ix.set_centroids(rng.standard_normal((len(sizes), d)).astype(np.float32))
    ix.set_codebooks(rng.standard_normal((M, 256, d // M)).astype(np.float32))
    for part in range(2):
        if part == 1:
            ix.reset()
        ln = rng.permutation(np.repeat(np.arange(len(sizes), dtype=np.int32), sizes))
        codes = rng.integers(0, 256, size=(len(ln), M), dtype=np.uint8)
        ids = rng.integers(-2**62, 2**62, size=len(ln), dtype=np.int64)
        half = len(ln) // 3
        for sl in (slice(0, half), slice(half, None)):
            if len(ln[sl]):
                ix.add_codes(ln[sl], codes[sl], ids[sl])
        for l in range(len(sizes)):
            c, i = ix.get_list(l)
            np.testing.assert_array_equal(c, codes[ln == l])
            np.testing.assert_array_equal(i, ids[ln == l])
