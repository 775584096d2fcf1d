"""From candidates to results of the exact indexes: the fused tail of fp32 lists (block and warp form),
its hand-over of lists that are too long, and the selection of long lists, at the edges of each."""
import numpy as np
import pytest

import oracle
from helpers import assert_exact
from indexsdk_b200 import datasets

pytestmark = pytest.mark.gpu
L2, IP = 1, 0


def _flat(b200, metric, xb, xq, k):
    ix = b200.IndexFlat(xb.shape[1], metric)
    ix.add(xb)
    D, I = ix.search(xq, k)
    Dr, Ir = oracle.flat_search(metric, xb, xq, k)
    assert_exact(D, I, Dr, Ir)
    return ix


# one-tile bases searched by many queries (a threshold over the whole base, the warp form up to k = 32), k on
# both sides of what a form takes, rows of 16 and of 32-float chunks
@pytest.mark.parametrize("metric", [L2, IP])
@pytest.mark.parametrize("n,d,nq,k", [(256, 64, 5000, 1), (40, 48, 20000, 2), (300, 128, 9000, 8), (2100, 64, 3000, 32),
                                      (2100, 80, 1500, 33), (5000, 64, 700, 100), (40000, 64, 40, 256), (40000, 64, 40, 257),
                                      (120000, 32, 3, 1000)])
def test_forms_of_the_tail(b200, metric, n, d, nq, k):
    _flat(b200, metric, datasets.gaussian(n, d, seed=1), datasets.gaussian(nq, d, seed=2), k)


@pytest.mark.parametrize("n,copies,k", [(200000, 1500, 10), (200000, 6000, 10), (9000, 1200, 5)])
def test_near_duplicates_outgrow_the_fused_tail(b200, n, copies, k):
    """`copies` rows closer together than the bf16 filter can tell apart: all survive the pruning."""
    xb = datasets.gaussian(n, 64, seed=1)
    near = xb[:1] + np.float32(1e-4) * datasets.gaussian(copies, 64, seed=3)
    xb[n - copies:] = near
    _flat(b200, L2, xb, np.concatenate([near[:2], datasets.gaussian(2, 64, seed=4)]), k)


@pytest.mark.parametrize("k", [1, 10, 129, 1024])
def test_ties_at_the_last_rank_go_to_the_lowest_positions(b200, k):
    """int8 rows of few distinct distances: thousands tie with the k-th key."""
    rng = np.random.default_rng(5)
    xb = rng.integers(-1, 2, size=(30000, 16)).astype(np.int8)
    xq = rng.integers(-1, 2, size=(9, 16)).astype(np.int8)
    for metric in (L2, IP):
        ix = b200.IndexInt8Flat(16, metric)
        ix.add(xb)
        D, I = ix.search(xq, k)
        Dr, Ir = oracle.int8_search(metric, xb, xq, k)
        assert_exact(D, I, Dr, Ir)


@pytest.mark.parametrize("keep", [0, 3, 40])
def test_filter_that_leaves_fewer_rows_than_k(b200, keep):
    """Fewer rows than k pass the filter of an int8 index large enough for a sampled threshold."""
    n, k = 150000, 10
    xb, xq = datasets.uniform_int8(n, 32, seed=1), datasets.uniform_int8(2, 32, seed=2)
    bits = np.zeros((2, n), bool)
    for q in range(2):
        bits[q, np.random.default_rng(q).permutation(n)[:keep]] = True
    for metric in (L2, IP):
        ix = b200.IndexInt8Flat(32, metric)
        ix.add(xb)
        D, I = ix.search_with_masks(xq, k, np.packbits(bits, axis=1, bitorder="little"))
        for q in range(2):
            rows = np.flatnonzero(bits[q])
            got = min(keep, k)
            assert (I[q, got:] == -1).all()
            if keep:
                Dr, Ir = oracle.int8_search(metric, xb[rows], xq[q:q + 1], got, labels=rows)
                assert_exact(D[q:q + 1, :got], I[q:q + 1, :got], Dr, Ir)


def _odd_queries(nq, d):
    xq = datasets.gaussian(nq, d, seed=7)
    one = [np.nan, np.inf, -np.inf, 1e15, 1e18, 1e20, 1e30, 3e38]
    whole = [1e18, 1e20, 3e38, 0.0, 1e-30, np.inf, np.nan]
    xq[np.arange(len(one)), 3] = one
    for i, v in enumerate(whole):
        xq[len(one) + i] = v
    return xq


# what the smallest base thresholds are taken from, one and several tiles, and larger ones
@pytest.mark.parametrize("metric", [L2, IP])
@pytest.mark.parametrize("n,d", [(1, 64), (40, 64), (300, 64), (2100, 80), (20000, 64)])
@pytest.mark.parametrize("rows", ["plain", "no number", "huge", "tiny", "equal"])
def test_without_an_error_bound_every_key_is_looked_at(b200, metric, n, d, rows):
    """Queries and rows whose norms overflow, vanish or are no numbers find what the search without thresholds
    finds (the entry point without allocations)."""
    import torch
    xb = datasets.gaussian(n, d, seed=n)
    if rows == "no number" and n > 20:
        xb[7], xb[9, 2], xb[11], xb[13] = np.inf, np.nan, -np.inf, 3e38
    elif rows == "huge":
        xb[n // 4:n // 2] = 3e19
    elif rows == "tiny":
        xb *= np.float32(1e-25)
    elif rows == "equal":
        xb[n // 2:] = xb[0]
    ix = b200.IndexFlat(d, metric)
    ix.add(xb)
    for nq, k in ((20, 1), (20, 10), (20, 300), (45, 100), (2000, 1)):
        if nq * ((n + 255) // 256 * 256) > 1 << 20:
            continue
        xq = _odd_queries(nq, d)
        xt = torch.from_numpy(xq).cuda()
        out = []
        for f in (ix.search_device, ix.search_device_noalloc):
            for q0 in range(0, nq, nq if f == ix.search_device else 1000):
                m = min(nq - q0, nq if f == ix.search_device else 1000)
                if q0 == 0:
                    D, I = torch.empty(nq, k, device="cuda"), torch.empty(nq, k, device="cuda", dtype=torch.int64)
                torch.cuda.synchronize()
                f(xt[q0:].data_ptr(), m, k, D[q0:].data_ptr(), I[q0:].data_ptr())
            torch.cuda.synchronize()
            out.append((D.cpu().numpy(), I.cpu().numpy()))
        np.testing.assert_array_equal(out[0][1], out[1][1])
        np.testing.assert_array_equal(out[0][0], out[1][0])


# both sides of the lines by number of queries: thresholds for bases of one tile (2^14 keys), the warp form
# (one query per SM up to k = 8, eight beyond)
@pytest.mark.parametrize("n,d,nq,k", [(40, 64, 409, 1), (40, 64, 410, 1), (256, 64, 63, 1), (256, 64, 64, 1), (5000, 64, 147, 8),
                                      (5000, 64, 148, 8), (5000, 64, 1183, 9), (5000, 64, 1184, 9)])
def test_lines_by_number_of_queries(b200, n, d, nq, k):
    _flat(b200, L2, datasets.gaussian(n, d, seed=1), datasets.gaussian(nq, d, seed=2), k)
