"""Multi-index search of small members with a threshold per (member, query): where it can go wrong
are members too small for a bound, members far apart in scale, rows that overflow their candidate
list (the group is then searched without thresholds), and infinite keys."""
import numpy as np
import pytest

import oracle
from helpers import assert_close_gap_aware, assert_exact
from indexsdk_b200 import datasets

pytestmark = pytest.mark.gpu
L2, IP = 1, 0


def _group(b200, kind, bases):
    is_int, metric = kind.startswith("i8"), 2 if kind.endswith("cos") else (IP if kind.endswith("ip") else L2)
    out = []
    for x in bases:
        if is_int:
            ix = b200.IndexInt8Flat(x.shape[1], metric)
        else:
            ix = b200.IndexFlat(x.shape[1], metric, dtype=b200.F16 if kind.startswith("f16") else b200.F32)
        ix.add(x)
        out.append(ix)
    ref = (lambda x, q, k: oracle.int8_search(metric, x, q, k)) if is_int else \
          (lambda x, q, k: oracle.flat_search(metric, x, q, k))
    return out, ref


def _check(b200, kind, bases, xq, k):
    ix, ref = _group(b200, kind, bases)
    D, I = b200.search_multi(ix, xq, k, merged=False)
    for i, x in enumerate(bases):
        Dr, Ir = ref(x, xq, k)
        if kind.startswith("f16"):
            # the library's bar for fp16 storage: sums of exact products in another order
            assert_close_gap_aware(D[i], I[i], Dr, Ir, 1e-3, f"member {i}")
        else:
            assert_exact(D[i], I[i], Dr, Ir)


# k against the rows: no bound at all (fewer bursts than k), a loose one, bursts of 8, bursts of 32
@pytest.mark.parametrize("kind", ["f32_l2", "f32_ip", "f16_l2", "f16_ip", "i8_l2", "i8_ip", "i8_cos"])
@pytest.mark.parametrize("d,nq,k,sizes", [(64, 1, 1, (1, 31, 32, 33, 257)),
                                          (128, 129, 10, (9, 90, 2561, 2560, 5000)),
                                          (256, 5, 100, (3201, 1100, 799, 12000, 40))])
def test_thresholds_at_the_edges(b200, kind, d, nq, k, sizes):
    if kind.startswith("i8"):
        bases = [datasets.uniform_int8(n, d, seed=i) for i, n in enumerate(sizes)]
        xq = datasets.uniform_int8(nq, d, seed=99)
    else:
        scale = [1.0, 0.01, 30.0, 1.0, 1.0] if kind == "f32_l2" else [1.0] * 5
        bases = [np.float32(scale[i]) * datasets.gaussian(n, d, seed=i) for i, n in enumerate(sizes)]
        xq = datasets.gaussian(nq, d, seed=99)
        if kind.startswith("f16"):
            bases, xq = [oracle.round_fp16(x) for x in bases], oracle.round_fp16(xq)
    _check(b200, kind, bases, xq, k)


@pytest.mark.parametrize("kind", ["f32_l2", "i8_ip"])
def test_overflow_is_searched_without_thresholds(b200, kind):
    """One member holds 3 000 copies of the same few rows: every key ties with the bound."""
    rng = np.random.default_rng(3)
    gen = datasets.uniform_int8 if kind.startswith("i8") else datasets.gaussian
    few = gen(4, 64, seed=1)
    bases = [gen(3000, 64, seed=2), few[rng.integers(0, 4, size=3000)]]
    _check(b200, kind, bases, gen(7, 64, seed=3), 10)


def test_infinite_distances_fill_up_a_short_member(b200):
    """Rows whose distance overflows to infinity still come after the finite ones."""
    x = datasets.gaussian(400, 64, seed=1)
    x[5:] = 3e19                                  # squared norm 5.8e40: not finite in fp32
    _check(b200, "f32_l2", [x, datasets.gaussian(700, 64, seed=2)], datasets.gaussian(3, 64, seed=3), 10)


@pytest.mark.parametrize("metric", [L2, IP])
def test_a_list_too_long_for_the_fused_tail_costs_its_own_kernels_only(b200, metric):
    """1 100 rows of one member closer together than the bf16 filter can tell apart all survive the pruning.
    The candidates are complete, so nothing has to be searched again: two kernels more (exact distances, order)
    than a call without such rows."""
    k, d = 100, 64
    rng = np.random.default_rng(5)
    plain = [datasets.gaussian(n, d, seed=i) for i, n in enumerate((12000, 9000, 11000))]
    near = plain[1].copy()
    near[rng.permutation(9000)[:1100]] = 3 * near[:1] + np.float32(1e-4) * datasets.gaussian(1100, d, seed=8)
    xq = datasets.gaussian(6, d, seed=9)
    xq[2] = 3 * near[0]
    launches = []
    for bases in (plain, [plain[0], near, plain[2]]):
        ix, ref = _group(b200, "f32_l2" if metric == L2 else "f32_ip", bases)
        b200.search_multi(ix, xq, k, merged=False)
        before = b200.search_multi_stats()["group_launches"]
        D, I = b200.search_multi(ix, xq, k, merged=False)
        launches.append(b200.search_multi_stats()["group_launches"] - before)
        for i, x in enumerate(bases):
            Dr, Ir = oracle.flat_search(metric, x, xq, k)
            assert_exact(D[i], I[i], Dr, Ir)
    assert launches[1] == launches[0] + 2


@pytest.mark.parametrize("metric", [L2, IP])
@pytest.mark.parametrize("nq,k", [(20, 1), (300, 10)])
def test_a_member_without_an_error_bound(b200, metric, nq, k):
    """A row with a NaN leaves a member's largest norm undefined; the other members' norms say nothing about
    its rows, of which one is near the largest float."""
    bases = [datasets.gaussian(n, 64, seed=i) for i, n in enumerate((1, 40, 300))]
    bases[1][7], bases[1][9, 2], bases[1][11], bases[1][13] = np.inf, np.nan, -np.inf, 3e38
    ix, _ = _group(b200, "f32_l2" if metric == L2 else "f32_ip", bases)
    xq = datasets.gaussian(nq, 64, seed=9)
    D, I = b200.search_multi(ix, xq, k, merged=False)
    for i in range(3):
        assert_exact(D[i], I[i], *ix[i].search(xq, k))     # few rows: every key is looked at


# members of one size, on both sides of the line for thresholds from every fourth tile (by queries: 8, 21, 43 bursts of 8 per k)
@pytest.mark.parametrize("kind", ["f32_l2", "f32_ip", "i8_l2", "f16_l2"])
@pytest.mark.parametrize("nq,k", [(1, 31), (1, 33), (64, 12), (64, 13), (130, 5), (130, 6)])
def test_thresholds_from_every_fourth_tile(b200, kind, nq, k):
    sizes = (8500, 8192, 8400)                   # 32 to 34 tiles: 256 bursts of 8 in every fourth
    gen = datasets.uniform_int8 if kind.startswith("i8") else datasets.gaussian
    bases, xq = [gen(n, 64, seed=i) for i, n in enumerate(sizes)], gen(nq, 64, seed=99)
    if kind.startswith("f16"):
        bases, xq = [oracle.round_fp16(x) for x in bases], oracle.round_fp16(xq)
    _check(b200, kind, bases, xq, k)
