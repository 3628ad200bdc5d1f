"""Which exact hubs the count pass takes in hash shares, and which go to tables
in global memory (many of several 100,000 neighbours)."""
import ctypes as C

import numpy as np
import pytest

import lpa_b200 as L
import oracle

REACH = 2048 << 12  # degrees the shares reach
BLOCKS = 296


def _limit(degrees, blocks=BLOCKS):
    d = np.asarray(degrees, np.uint32)
    f = L.lib().lpa_test_hash_share_limit
    f.restype = C.c_uint64
    return f(d.ctypes.data_as(C.POINTER(C.c_uint32)), C.c_size_t(len(d)), blocks)


@pytest.mark.parametrize("degrees,limit", [
    ([], REACH),
    ([2048], REACH),
    ([1000000], REACH),
    ([1000000] * 10, REACH),         # 6.7 ms in shares, 6.2 to 22 in tables
    ([1000000] * 100, 2047),         # 60 ms against 6 to 38
    ([300000] * 300, 2047),          # 28 ms against 5.5 to 38
    ([100000] * 1000, REACH),        # 8.4 to 23 ms against 3.0 to 27
    ([30000] * 2000, REACH),
    ([3000] * 50 + [1000000] * 100, 3000),
    ([REACH + 1], REACH),            # beyond the shares' reach: tables whatever the rest
    ([REACH + 1] + [5000] * 100, REACH),
])
def test_limit(degrees, limit):
    assert _limit(degrees) == limit
    assert _limit(np.random.default_rng(0).permutation(np.asarray(degrees, np.uint32))) == limit


@pytest.mark.gpu
@pytest.mark.parametrize("budget", [0, 96 << 20], ids=["resident", "streamed"])
@pytest.mark.parametrize("variant", [None, L.Variant.TWO_PASS], ids=["fixed", "two_pass"])
def test_hubs_in_tables(variant, budget):
    rng = np.random.default_rng(2)
    n, hubs, d = 600000, 64, 400000
    lists = [np.flatnonzero(rng.random(n, np.float32) < d / n).astype(np.uint32) for _ in range(hubs)]
    lists.append(np.arange(3000, dtype=np.uint32) * 7)
    deg = np.ones(n, np.int64)
    deg[:len(lists)] = [len(x) for x in lists]
    row = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint64)
    clm = np.concatenate(lists + [rng.integers(0, n, n - len(lists)).astype(np.uint32)])
    assert _limit(deg[deg > 2047]) < 300000
    hist, changed = oracle.lp_run(row, clm, 3, 0, 1)
    g = L.HostGraph.from_csr(row, clm).compress(0, 128)
    opts = dict(stream_budget=budget)
    if variant is not None:
        opts.update(dispatch=L.Dispatch.FORCE, force_variant=int(variant))
    for refused in (None, b"global count tables"):  # without memory for tables: shares
        L.lib().lpa_test_refuse(refused)
        try:
            p = L.Propagator(g, **opts)
        finally:
            L.lib().lpa_test_refuse(None)
        with p:
            for it in range(3):
                assert p.iterate() == changed[it]
                assert np.array_equal(p.labels(), hist[it])
