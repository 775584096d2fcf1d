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


def test_indexes_share_the_spare_arrays_of_their_merges(b200):
    """Reloading an index leaves a set of list arrays and work arrays behind.  They belong to the device, not to
    the index, and go with the last index."""
    import torch
    n, M, nlist = 400000, 16, 16
    rng = np.random.default_rng(3)
    ln = rng.integers(0, nlist, size=n).astype(np.int32)
    codes = rng.integers(0, 256, size=(n, M), dtype=np.uint8)
    ids = np.arange(n, dtype=np.int64)
    cent, cb = rng.standard_normal((nlist, M)).astype(np.float32), rng.standard_normal((M, 256, 1)).astype(np.float32)

    def loaded():
        ix = b200.IndexIVFPQ(M, nlist, M, 8, by_residual=False)
        ix.set_centroids(cent)
        ix.set_codebooks(cb)
        for _ in range(2):
            ix.reset()
            ix.add_codes(ln, codes, ids)
        return ix

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    loaded()                                    # kernels and the runtime's own memory
    first = free()
    held = [loaded(), loaded()]
    two = free()
    held += [loaded() for _ in range(8)]
    own = (two - free()) / 8
    # lists (16 + 8 + 4 bytes a vector) and the staging of add_codes (16 + 8 + 4 + 4), each with a quarter of spare room
    assert own < 1.25 * n * (28 + 32) + (6 << 20)
    np.testing.assert_array_equal(np.sort(held[3].get_list(5)[1]), ids[ln == 5])
    del held
    assert first - free() < 16 << 20
