"""Host threads sharing one index handle.

The reference lets several threads search one index when MX_INDEX_MULTITHREAD=1
(feature_retrieval/src/ascendfaiss/ascend/impl/AscendIndexImpl.h:62,230: shared lock for search).
An index here owns one stream and one set of scratch buffers, so the C ABI serialises the calls on
a handle; the test runs searches of different sizes from several threads at once (ctypes releases
the GIL during the call) and compares every result with the single-threaded one.
"""
import os
import subprocess
import threading

import numpy as np
import pytest

from indexsdk_b200 import datasets

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _hammer(index, queries, k, expect, errors, rounds):
    try:
        for _ in range(rounds):
            for xq, (Dr, Ir) in zip(queries, expect):
                D, I = index.search(xq, k)
                if not (np.array_equal(I, Ir) and np.array_equal(D.view(np.uint32), Dr.view(np.uint32))):
                    errors.append("result differs from the single-threaded search")
                    return
    except Exception as e:  # noqa: BLE001 - reported to the main thread
        errors.append(repr(e))


def test_concurrent_searches_on_one_flat_index(b200):
    d, k = 64, 10
    ix = b200.IndexFlat(d, b200.METRIC_L2)
    ix.add(datasets.gaussian(30000, d, seed=0))
    # different batch sizes: scratch buffers would be re-sized under a concurrent reader
    queries = [datasets.gaussian(n, d, seed=10 + n) for n in (3, 200, 17, 900)]
    expect = [ix.search(xq, k) for xq in queries]
    errors = []
    threads = [threading.Thread(target=_hammer, args=(ix, queries[i:] + queries[:i], k, expect[i:] + expect[:i], errors, 6))
               for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[:3]


def test_concurrent_searches_on_one_ivfpq_index(b200):
    d, nlist, M, k = 64, 64, 16, 10
    xb, _ = datasets.mixture(20000, d, nlist, seed=4)
    cent, cb = datasets.train_ivfpq(xb[:4000], nlist, M, True, niter=3)
    ix = b200.IndexIVFPQ(d, nlist, M, 8, by_residual=True)
    ix.set_centroids(cent)
    ix.set_codebooks(cb)
    ix.add(xb)
    ix.nprobe = 8
    queries = [datasets.mixture(n, d, nlist, seed=20 + n, centers_seed=4)[0] for n in (5, 1300, 64)]
    expect = [ix.search(xq, k) for xq in queries]
    errors = []
    threads = [threading.Thread(target=_hammer, args=(ix, queries[i:] + queries[:i], k, expect[i:] + expect[:i], errors, 4))
               for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[:3]


@pytest.mark.parametrize("which", ["select", "finish", "bound"])
def test_two_indexes_share_their_kernels(b200, which):
    """Calls on different handles run concurrently, also when the same kernels need another amount of
    shared memory in each: what one thread asks for must not shrink what the other was granted.  (Threads of
    a C++ program: the window is too short for threads that take turns at the interpreter.)"""
    src = os.path.join(ROOT, "tests", "cpp", "test_two_indexes.cpp")
    build = os.path.join(ROOT, "indexsdk_b200", "_build")
    exe = os.path.join(build, "test_two_indexes")
    if not os.path.exists(exe) or os.path.getmtime(src) > os.path.getmtime(exe):
        subprocess.run(["/usr/bin/g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "include"), src, "-o", exe,
                        "-L", build, "-lb200idx", "-Wl,-rpath," + build, "-lpthread"], check=True)
    r = subprocess.run([exe, which], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "0 failed" in r.stdout, r.stdout[-2000:] + r.stderr[-2000:]


def test_statistics_are_read_between_searches_not_inside_them(b200):
    """A thread that asks for the statistics while another searches sees whole searches: the codes visited
    belong to the queries counted, in between and at the end."""
    d, nlist, M, k, n = 32, 16, 8, 10, 20000
    rng = np.random.default_rng(4)
    ix = b200.IndexIVFPQ(d, nlist, M, 8, by_residual=False)
    ix.set_centroids(datasets.gaussian(nlist, d, seed=2))
    ix.set_codebooks(rng.standard_normal((M, 256, d // M)).astype(np.float32))
    ix.add_codes(rng.integers(0, nlist, size=n).astype(np.int32), rng.integers(0, 256, size=(n, M), dtype=np.uint8))
    ix.nprobe = nlist                                          # every query visits every vector
    xq = datasets.gaussian(40000, d, seed=1)                   # three pages
    stop, wrong = threading.Event(), []

    def watch():
        while not stop.is_set():
            s = ix.stats()
            if s["scan_codes"] != s["queries"] * n:
                wrong.append((s["queries"], s["scan_codes"]))

    t = threading.Thread(target=watch)
    t.start()
    for _ in range(8):
        ix.search(xq, k)
    stop.set()
    t.join()
    s = ix.stats()
    assert s["queries"] == 8 * len(xq) and s["scan_codes"] == s["queries"] * n
    assert not wrong, wrong[:3]
