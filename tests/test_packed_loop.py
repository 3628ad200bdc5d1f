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
