"""Performance cases: what users of the library have it do, through its public entry points.

A case is a dict of plain values.  ``prepare`` makes what a program holds before the call -- the
loaded index and the queries --, ``run`` is one pass through the entry point and returns its whole
result, ``work`` counts what no implementation can do without, ``tolerance`` says how far a correct
implementation's result may be off.  All inputs are seeded and synthetic.

kind   : flat | int8 | ivfpq | multi | build
api    : host (numpy arrays in and out, the call most programs make) | device (addresses of
         tensors that already live on the GPU)
"""
import math

import numpy as np
import torch

import indexsdk_b200 as b

METRICS = {"ip": b.METRIC_INNER_PRODUCT, "l2": b.METRIC_L2, "cos": b.METRIC_INT8_COSINE}
DTYPES = {"f32": b.F32, "f16": b.F16}
CHUNK = 1_000_000          # vectors generated and added at a time


def listed():
    return [
        # One query against a mid-sized gallery, as an online service asks it: latency is all that counts.
        dict(name="flat_f32_single", kind="flat", dtype="f32", metric="l2", n=100_003, d=128, nq=1, k=10,
             api="host", masked=False),
        # The exact-search benchmark: 1 M x 128 fp32, a batch of 1024 queries, k = 100.
        dict(name="flat_f32_1m", kind="flat", dtype="f32", metric="l2", n=1_000_000, d=128, nq=1024, k=100,
             api="device", masked=False),
        # fp16 storage (the default of the C++ classes), L2, face-feature sizes, a ragged ordinary batch.
        dict(name="flat_f16_ragged", kind="flat", dtype="f16", metric="l2", n=300_007, d=512, nq=100, k=10,
             api="host", masked=False),
        # Large-k batch search of one 2.5 M x 768 fp16 inner-product index: one GPU's part of the
        # multi-index benchmark, the largest amount of arithmetic here.
        dict(name="flat_f16_large_k", kind="flat", dtype="f16", metric="ip", n=2_500_000, d=768, nq=4096, k=1000,
             api="device", masked=False),
        # The int8 benchmark: 4 M x 256, inner product, 256 queries, k = 100.
        dict(name="int8_4m", kind="int8", metric="ip", n=4_000_000, d=256, nq=256, k=100, api="device", masked=False),
        # int8 L2 with a per-query filter over the base (search_with_masks), odd sizes.
        dict(name="int8_masked_ragged", kind="int8", metric="l2", n=200_003, d=512, nq=33, k=10, api="host",
             masked=True),
        # The IVFPQ benchmark: 10 M x 128, 16384 lists, 16-byte residual codes, nprobe 64, k = 10, 10 000 queries.
        dict(name="ivfpq_10m", kind="ivfpq", n=10_000_000, d=128, nlist=16384, M=16, residual=True, nprobe=64, k=10,
             nq=10_000, sigma=0.1, skew=0.0, api="device"),
        # One online query against an IVFPQ index of ordinary size, lists of uneven length.
        dict(name="ivfpq_single", kind="ivfpq", n=1_000_000, d=128, nlist=4096, M=32, residual=True, nprobe=32, k=10,
             nq=1, sigma=0.5, skew=0.5, api="host"),
        # Wide codes and a large k: 48-byte codes of 96 dimensions, nprobe 128, k = 100 (the 100 M
        # configuration's parameters on a base of 5 M).
        dict(name="ivfpq_wide", kind="ivfpq", n=5_000_000, d=96, nlist=16384, M=48, residual=True, nprobe=128, k=100,
             nq=1000, sigma=0.5, skew=0.5, api="device"),
        # Short codes of raw vectors, few long lists, k = 300, a batch of 64: the sizes of the
        # reference's IVFPQ latency target (nlist 1024, d 128, M 4, k 300, 10 M vectors).
        dict(name="ivfpq_short_raw", kind="ivfpq", n=10_000_000, d=128, nlist=1024, M=4, residual=False, nprobe=64,
             k=300, nq=64, sigma=0.5, skew=0.5, api="host"),
        # Many small indexes searched together and merged (one per tenant or camera).
        dict(name="multi_small", kind="multi", dtype="f32", metric="l2", indexes=32, n=20_011, d=128, nq=64, k=10,
             merged=True),
        # Loading an IVFPQ index: assignment, encoding, list building, and the lists read back (what
        # copying a built index to the CPU does).
        dict(name="ivfpq_build", kind="build", n=300_000, d=128, nlist=256, M=16, residual=True, sigma=0.5, skew=0.5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges that the listed ones span."""
    kind = rng.choice(["flat", "flat", "flat", "int8", "int8", "ivfpq", "ivfpq", "ivfpq", "multi", "build"])
    d = rng.choice([64, 96, 128, 128, 256, 384, 512, 768])
    if kind in ("flat", "int8"):
        c = dict(kind=kind, metric=rng.choice(["ip", "l2"] if kind == "flat" else ["ip", "l2", "cos"]), d=d,
                 n=_log(rng, 10_000, 4_000_000 if kind == "int8" else 2_500_000), k=_log(rng, 1, 1000),
                 api=rng.choice(["host", "device"]), masked=rng.random() < 0.2)
        if kind == "flat":
            c["dtype"] = rng.choice(["f32", "f16"])
        c["nq"] = _log(rng, 1, max(1, min(4096, int(8e12 / (2.0 * c["n"] * d)))))
        if c["masked"]:
            c["api"] = "host"
            c["nq"] = max(1, min(c["nq"], 32_000_000 // c["n"]))
        return c
    if kind == "multi":
        nx = _log(rng, 4, 64)
        dtype = rng.choice(["f32", "f16", "int8"])
        return dict(kind=kind, dtype=dtype, metric=rng.choice(["ip", "l2"]), indexes=nx,
                    n=_log(rng, 1000, min(50_000, 1_000_000 // nx)), d=min(d, 512), nq=_log(rng, 1, 128),
                    k=_log(rng, 1, 100), merged=rng.random() < 0.7)
    d, M = rng.choice([(128, 16), (128, 16), (128, 32), (128, 4), (128, 8), (96, 48), (64, 16), (128, 64), (64, 32)])
    common = dict(kind=kind, d=d, M=M, residual=rng.random() < 0.7, sigma=rng.choice([0.1, 0.5, 0.5, 1.0]),
                  skew=rng.choice([0.0, 0.5]))
    if kind == "build":
        return dict(common, n=_log(rng, 20_000, 400_000), nlist=_log(rng, 64, 512))
    nlist = _log(rng, 256, 16384)
    c = dict(common, nlist=nlist, n=_log(rng, max(100_000, 40 * nlist), 10_000_000), k=_log(rng, 1, 300),
             nprobe=_log(rng, 1, min(128, nlist // 4)), api=rng.choice(["host", "device"]))
    # vectors visited: no more than the listed cases of the same code width
    limit = 6.2e9 / M if M >= 16 else 4e7
    c["nq"] = _log(rng, 1, max(1, min(10_000, int(limit / (c["nprobe"] * c["n"] / nlist)))))
    return c


# ---- inputs ----
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _rows(kind, metric, n, d, g):
    """Base rows or queries of an exact index: N(0, 1) floats (unit length for inner products) or
    int8 uniform in [-128, 127]."""
    if kind == "int8":
        return torch.randint(-128, 128, (n, d), generator=g, device="cuda", dtype=torch.int8)
    x = torch.randn(n, d, generator=g, device="cuda")
    if metric == "ip":
        x /= x.norm(dim=1, keepdim=True)
    return x


def _exact_index(kind, dtype, metric, n, d, g):
    ix = b.IndexInt8Flat(d, METRICS[metric]) if kind == "int8" else b.IndexFlat(d, METRICS[metric], DTYPES[dtype])
    for lo in range(0, n, CHUNK):
        x = _rows(kind, metric, min(CHUNK, n - lo), d, g)
        torch.cuda.synchronize()
        ix.add_device(x.data_ptr(), x.shape[0])
    return ix


class _Mixture:
    """Gaussian mixture with one component per list: centres ~ N(0, 1), points = centre +
    N(0, sigma^2), component weights log-normal with spread `skew`.  The centres are the coarse
    centroids; the codebooks are a few k-means iterations on a sample of what is encoded."""

    def __init__(self, case, seed):
        self.case, self.g = case, _gen(seed)
        self.centres = torch.randn(case["nlist"], case["d"], generator=self.g, device="cuda")
        w = torch.exp(case["skew"] * torch.randn(case["nlist"], generator=self.g, device="cuda"))
        self.cdf = torch.cumsum(w / w.sum(), 0)

    def points(self, n):
        u = torch.rand(n, generator=self.g, device="cuda")
        which = torch.searchsorted(self.cdf, u).clamp_(max=self.case["nlist"] - 1)
        x = torch.randn(n, self.case["d"], generator=self.g, device="cuda")
        return x.mul_(self.case["sigma"]).add_(self.centres[which]), which

    def index(self):
        c = self.case
        ix = b.IndexIVFPQ(c["d"], c["nlist"], c["M"], 8, by_residual=c["residual"])
        ix.set_centroids(self.centres.cpu().numpy())
        x, which = self.points(16384)
        if c["residual"]:
            x = x - self.centres[which]
        x = x.cpu().numpy()
        ds = c["d"] // c["M"]
        ix.set_codebooks(np.stack([b.kmeans(x[:, m * ds:(m + 1) * ds], 256, 4, m) for m in range(c["M"])]))
        return ix


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind in ("flat", "int8"):
        g = _gen(seed)
        st["ix"] = _exact_index(kind, case.get("dtype"), case["metric"], case["n"], case["d"], g)
        xq = _rows(kind, case["metric"], case["nq"], case["d"], g)
        if case["masked"]:
            keep = torch.rand(case["nq"], case["n"], generator=g, device="cuda") < 0.5
            st["mask"] = np.packbits(keep.cpu().numpy(), axis=1, bitorder="little")
    elif kind == "multi":
        g = _gen(seed)
        ekind = "int8" if case["dtype"] == "int8" else "flat"
        st["ix"] = [_exact_index(ekind, case["dtype"], case["metric"], case["n"] + 7 * i, case["d"], g)
                    for i in range(case["indexes"])]
        xq = _rows(ekind, case["metric"], case["nq"], case["d"], g)
    else:
        mix = _Mixture(case, seed)
        ix = st["ix"] = mix.index()
        if kind == "build":
            st["x"] = mix.points(case["n"])[0]
            torch.cuda.synchronize()
            return st
        for lo in range(0, case["n"], CHUNK):
            x = mix.points(min(CHUNK, case["n"] - lo))[0]
            torch.cuda.synchronize()
            ix.add_device(x.data_ptr(), x.shape[0])
        ix.nprobe = case["nprobe"]
        xq = mix.points(case["nq"])[0]
    if case.get("api") == "device":
        st["xq"] = xq
        st["D"] = torch.empty(case["nq"], case["k"], device="cuda")
        st["I"] = torch.empty(case["nq"], case["k"], device="cuda", dtype=torch.int64)
    else:
        st["xq"] = xq.cpu().numpy()
    torch.cuda.synchronize()
    return st


def run(st):
    case, ix = st["case"], st["ix"]
    if case["kind"] == "build":
        ix.reset()
        ix.add_device(st["x"].data_ptr(), case["n"])
        lists = [ix.get_list(i) for i in range(case["nlist"])]
        return np.concatenate([codes for codes, _ in lists]), np.concatenate([ids for _, ids in lists])
    if case["kind"] == "multi":
        return b.search_multi(ix, st["xq"], case["k"], merged=case["merged"])
    if case.get("masked"):
        return ix.search_with_masks(st["xq"], case["k"], st["mask"])
    if case["api"] == "host":
        return ix.search(st["xq"], case["k"])
    ix.search_device(st["xq"].data_ptr(), case["nq"], case["k"], st["D"].data_ptr(), st["I"].data_ptr())
    return st["D"], st["I"]


def work(case):
    """Every base row (or probed code), query and centroid read once in its stored type, results
    written once; multiply-adds of the distances as two operations, a table lookup's addition as one."""
    kind, n, d = case["kind"], case["n"], case["d"]
    if kind in ("flat", "int8", "multi"):
        rows = sum(n + 7 * i for i in range(case["indexes"])) if kind == "multi" else n
        elem = 1 if kind == "int8" or case["dtype"] == "int8" else (2 if case["dtype"] == "f16" else 4)
        nq, k = case["nq"], case["k"]
        outs = case["indexes"] if kind == "multi" and not case["merged"] else 1
        nbytes = rows * d * elem + nq * d * elem + outs * nq * k * 12 + (nq * n // 8 if case.get("masked") else 0)
        return dict(bytes=float(nbytes), flops=2.0 * rows * d * nq)
    nlist, M = case["nlist"], case["M"]
    if kind == "build":
        # assignment to the nearest of nlist centroids, M searches of 256 codewords; codes and ids out
        return dict(bytes=float(n * d * 4 + nlist * d * 4 + n * (M + 8)), flops=2.0 * n * d * (nlist + 256))
    nq, k = case["nq"], case["k"]
    visited = nq * case["nprobe"] * n / nlist
    nbytes = min(float(n), visited) * M + nlist * d * 4 + nq * d * 4 + nq * k * 12
    return dict(bytes=nbytes, flops=2.0 * nq * nlist * d + 2.0 * nq * 256 * d + visited * M)


def tolerance(case):
    """fp32 and int8 indexes and IVFPQ return distances of a defined summation order and break ties
    by id: exact.  fp16 storage: fp32 sums of exact products in any order (against 64-bit sums: 9e-7
    over all distances, 2.3e-6 the worst, 0.15 % of the ids at k = 1000); ranks closer than that
    may swap."""
    if case.get("dtype") == "f16":
        return {"rel": 4e-6, "max": 1e-5, "differ": 0.006}
    return "exact"
