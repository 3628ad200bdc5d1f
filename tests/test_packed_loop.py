"""lpa_run of plans that are all lane-per-vertex chunks: one cooperative launch."""
import ctypes as C

import numpy as np
import pytest

import lpa_b200 as L
import oracle

pytestmark = pytest.mark.gpu


def test_barrier_gives_up():
    """The loop's barrier is bounded by a time, and the handle outlives running out of it."""
    g = L.HostGraph.road(200, 301, seed=7)
    row, clm = g.csr()
    g.compress(0, 128)
    hist, _ = oracle.lp_run(row, clm, 25, 0, 1)
    with L.Propagator(g) as p:
        L.lib().lpa_test_loop_wait(p._h, C.c_uint64(0))
        with pytest.raises(L.LpaError) as e:
            p.run(25)
        assert e.value.status == L.Status.TIMEOUT
        L.lib().lpa_test_loop_wait(p._h, C.c_uint64(60 * 10**9))
        p.init_labels()
        assert p.run(25) == 25
        assert np.array_equal(p.labels(), hist[24])


def _tiny_lists(n, seed):
    """Lists of 0 to 15 ids, a third of them with runs of consecutive ones."""
    rng = np.random.default_rng(seed)
    lists = []
    for v in range(n):
        d = int(rng.integers(0, 16))
        if v % 3 or d < 5:
            ids = np.unique(rng.integers(0, n, d))
        else:
            start = int(rng.integers(0, n - 4))
            ids = np.unique(np.concatenate([np.arange(start, start + 4), rng.integers(0, n, d - 4)]))
        lists.append(ids.astype(np.uint32))
    row = np.concatenate([[0], np.cumsum([len(x) for x in lists])]).astype(np.uint64)
    return row, np.concatenate(lists)


@pytest.mark.parametrize("iters", [4, 7])
@pytest.mark.parametrize("thresh", [0, 6, 16])
@pytest.mark.parametrize("graph", ["tiny", "road"])
def test_whole_runs(graph, thresh, iters):
    """Degrees up to 15 in the stream and the small CSR (walked and counted in the
    label slots above 8), and more chunks than resident warps; after an odd
    number of iterations too.  Then the captured loop, for a grid that does not fit."""
    if graph == "tiny":
        row, clm = _tiny_lists(9999, thresh)
        g = L.HostGraph.from_csr(row, clm)
    else:
        g = L.HostGraph.road(1404, 331, seed=3)  # 14,500 chunks
        row, clm = g.csr()
    g.compress(thresh, 128)
    hist, changed = oracle.lp_run(row, clm, iters, 0, 1)
    with L.Propagator(g) as p:
        launches = p.stats().launches
        assert p.run(iters) == iters
        assert p.stats().launches == launches + 1
        assert np.array_equal(p.labels(), hist[-1])
        assert list(p.changed_history(iters)) == changed
        p.init_labels()
        L.lib().lpa_test_refuse(b"packed loop")
        try:
            assert p.run(iters) == iters
        finally:
            L.lib().lpa_test_refuse(None)
        assert p.stats().launches > launches + iters
        assert np.array_equal(p.labels(), hist[-1])
        assert list(p.changed_history(iters)) == changed
