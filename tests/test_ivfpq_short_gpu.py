"""IVFPQ search of short codes (M = 4 and 8): bound, collection and exact order against the oracle.
Where it can go wrong: k against what the nearest lists hold, lists shorter than a block's unit or
empty, ties that outgrow the sort (2 048 pairs) and the candidate row (32 768), duplicate-free
ordering by label, several shares per query."""
import numpy as np
import pytest

import oracle
from helpers import assert_exact
from indexsdk_b200 import datasets

pytestmark = pytest.mark.gpu


def _check(b200, xb, ids, cent, cb, resid, xq, nprobe, k):
    nlist, M = cent.shape[0], cb.shape[0]
    ix = b200.IndexIVFPQ(xb.shape[1], nlist, M, 8, by_residual=resid)
    ix.set_centroids(cent)
    ix.set_codebooks(cb)
    ix.add_with_ids(xb, ids)
    ix.nprobe = nprobe
    D, I = ix.search(xq, k)
    ln = oracle.ivf_assign(cent, xb)
    off, cs, idl = oracle.build_lists(ln, oracle.pq_encode(cb, xb, resid, cent, ln), ids, nlist)
    Dr, Ir = oracle.ivfpq_search(cent, cb, resid, off, cs, idl, xq, nprobe, k)
    assert_exact(D, I, Dr, Ir)
    return ix


@pytest.mark.parametrize("resid", [False, True])
@pytest.mark.parametrize("M,d,nlist,n,nq,nprobe,k", [
    (4, 64, 16, 3000, 1, 16, 1),           # one query, many shares of it
    (4, 128, 8, 40000, 3, 8, 300),
    (8, 64, 512, 5000, 70, 40, 100),       # lists of about ten vectors, some empty
    (8, 128, 8, 33000, 5, 5, 1024),
    (4, 64, 4, 900, 2, 2, 1024),           # fewer vectors than k
    (8, 96, 1300, 2600, 9, 1024, 10),      # the largest number of staged probes
])
def test_short_codes_vs_oracle(b200, resid, M, d, nlist, n, nq, nprobe, k):
    xb, _ = datasets.mixture(n, d, max(nlist // 3, 4), seed=4)
    xq, _ = datasets.mixture(nq, d, max(nlist // 3, 4), seed=5, centers_seed=4)
    rng = np.random.default_rng(1)
    ids = rng.permutation(n).astype(np.int64) * 3 - 1000     # unordered, some negative
    cent, cb = datasets.train_ivfpq(xb[:8000], min(nlist, 512), M, resid, niter=3)
    if nlist > 512:                                          # more lists than were trained: shifted copies
        cent = np.concatenate([cent + np.float32(0.01 * i) for i in range(3)])[:nlist]
    _check(b200, xb, ids, cent, cb, resid, xq, nprobe, k)


@pytest.mark.parametrize("resid", [False, True])
@pytest.mark.parametrize("copies", [3000, 40000])
def test_ties_beyond_the_sort_and_beyond_the_row(b200, resid, copies):
    """`copies` equal vectors in one list: the labels decide.  40 000 do not fit a candidate row, which
    residual encoding answers with the exact scan and raw encoding with a bound on the labels."""
    d, M, nlist, k = 64, 4, 4, 50
    xb, _ = datasets.mixture(2000, d, 4, seed=4)
    cent, cb = datasets.train_ivfpq(xb, nlist, M, resid, niter=3)
    xb = np.concatenate([xb, np.repeat(xb[:1], copies, axis=0)])
    ids = np.random.default_rng(2).permutation(len(xb)).astype(np.int64) - 500
    ix = _check(b200, xb, ids, cent, cb, resid, xb[:3], 4, k)
    assert (ix.stats()["fallback_queries"] > 0) == (copies == 40000 and resid)


def test_queries_that_hold_nan_or_infinity_find_what_the_exact_scan_finds(b200, monkeypatch):
    d, M, nlist = 64, 8, 8
    xb, _ = datasets.mixture(4000, d, 8, seed=4)
    cent, cb = datasets.train_ivfpq(xb, nlist, M, False, niter=3)
    xq = xb[:4].copy()
    xq[1, 3], xq[2, 5], xq[3] = np.nan, np.inf, 1e30
    out = []
    for exact in ("0", "1"):
        monkeypatch.setenv("B200IDX_IVFPQ_EXACT", exact)
        ix = b200.IndexIVFPQ(d, nlist, M, 8, by_residual=False)
        ix.set_centroids(cent)
        ix.set_codebooks(cb)
        ix.add(xb)
        ix.nprobe = 4
        out.append(ix.search(xq, 20))
    assert_exact(out[0][0], out[0][1], out[1][0], out[1][1])


@pytest.mark.parametrize("M,d,k", [(4, 64, 300), (8, 64, 20), (16, 64, 60), (48, 96, 100)])
def test_residual_queries_beyond_the_range_of_floats_find_what_the_exact_scan_finds(b200, monkeypatch, M, d, k):
    """With a component or a norm that overflows, |q - c|^2 + t2 - 2 q.cb can be NaN where the canonical distance
    is infinite."""
    nlist = 8
    xb, _ = datasets.mixture(4000, d, 8, seed=4)
    cent, cb = datasets.train_ivfpq(xb, nlist, M, True, niter=3)
    xq = xb[:9].copy()
    xq[1, 3], xq[2, 5], xq[3] = np.nan, np.inf, 1e30
    xq[4], xq[5, 7], xq[6] = 1e18, 3e38, np.inf
    xq[7, 1], xq[8, 2] = -1e19, 1e19
    out = []
    for exact in ("0", "1"):
        monkeypatch.setenv("B200IDX_IVFPQ_EXACT", exact)
        ix = b200.IndexIVFPQ(d, nlist, M, 8, by_residual=True)
        ix.set_centroids(cent)
        ix.set_codebooks(cb)
        ix.add(xb)
        ix.nprobe = nlist
        out.append(ix.search(xq, k))
    assert_exact(out[0][0], out[0][1], out[1][0], out[1][1])


# short codes: the distances that come with the probes are not what decides; wide codes scan with them
@pytest.mark.parametrize("M,d,k,how", [(4, 64, 10, "reversed"), (4, 64, 10, "zero"), (8, 64, 300, "zero"), (8, 64, 10, "nan"),
                                       (16, 64, 60, "reversed"), (16, 64, 60, "some"), (8, 64, 10, "some"), (64, 64, 300, "reversed")])
def test_given_probes_in_any_order(b200, M, d, k, how):
    import torch
    nlist, nprobe, nq = 32, 20, 50
    xb, _ = datasets.mixture(30000, d, nlist, seed=4, sigma=0.5)
    cent, cb = datasets.train_ivfpq(xb[:6000], nlist, M, True, niter=2)
    ix = b200.IndexIVFPQ(d, nlist, M, 8, by_residual=True)
    ix.set_centroids(cent)
    ix.set_codebooks(cb)
    ix.add(xb)
    ix.nprobe = nprobe
    xq = torch.from_numpy(datasets.mixture(nq, d, nlist, seed=5, centers_seed=4, sigma=0.5)[0]).cuda()
    cD = torch.empty(nq, nprobe, device="cuda")
    cI = torch.empty(nq, nprobe, device="cuda", dtype=torch.int64)
    D, I = torch.empty(nq, k, device="cuda"), torch.empty(nq, k, device="cuda", dtype=torch.int64)
    ix.coarse_device(xq.data_ptr(), nq, cD.data_ptr(), cI.data_ptr())
    if how == "some":                       # every other probe is none, the last one too
        cI[:, 1::2] = -1
        cD[:, 1::2] = float("nan")
    lists = cI.cpu().numpy()
    if how == "reversed":
        cD, cI = cD.flip(1).contiguous(), cI.flip(1).contiguous()
    elif how == "zero":
        cD.zero_()
    elif how == "nan":
        cD.fill_(float("nan"))
    torch.cuda.synchronize()
    ix.search_preassigned_device(xq.data_ptr(), nq, k, cD.data_ptr(), cI.data_ptr(), D.data_ptr(), I.data_ptr())
    ln = oracle.ivf_assign(cent, xb)
    codes = oracle.pq_encode(cb, xb, True, cent, ln)
    for q in range(0, nq, 7):               # the oracle over the vectors of the given lists
        rows = np.flatnonzero(np.isin(ln, lists[q]))
        off, cs, ids = oracle.build_lists(ln[rows], codes[rows], rows.astype(np.int64), nlist)
        Dr, Ir = oracle.ivfpq_search(cent, cb, True, off, cs, ids, xq[q:q + 1].cpu().numpy(), nlist, k)
        assert_exact(D[q:q + 1].cpu().numpy(), I[q:q + 1].cpu().numpy(), Dr, Ir)
