"""Plans that the device has no memory for: the call says so, the handle goes on
with the plan it had (or with the kernels that need less), and the labels stay
right.  lpa_test_refuse makes allocations fail by name."""
import contextlib

import numpy as np
import pytest
import torch

import lpa_b200 as L
import oracle

pytestmark = pytest.mark.gpu

CMS = 1024


@contextlib.contextmanager
def refuse(name):
    L.lib().lpa_test_refuse(name.encode())
    try:
        yield
    finally:
        L.lib().lpa_test_refuse(None)


@pytest.fixture(scope="module")
def case():
    g = L.HostGraph.rmat(15, 16, seed=5)
    row, clm = g.csr()
    assert np.diff(row).max() > 4096  # hubs, above the block table too
    g.compress(16, 128)
    return g, {cms: oracle.lp_run(row, clm, 6, cms, 1) for cms in (0, CMS)}


def _check(p, hist, changed, it):
    assert p.iterate() == changed[it]
    assert np.array_equal(p.labels(), hist[it])


@pytest.mark.parametrize("cms", [0, CMS])
@pytest.mark.parametrize("budget", [0, 4 << 20], ids=["resident", "streamed"])
@pytest.mark.parametrize("name", ["work items", "decode groups", "record groups", "count items", "count block items",
                                  "packed chunks", "two-pass scratch", "position index", "segment records"])
def test_failed_switch(case, name, budget, cms):
    g, want = case
    hist, changed = want[cms]
    if budget and name not in ("two-pass scratch", "position index", "segment records", "record groups"):
        name = "range " + name
    with L.Propagator(g, cms_threshold=cms, stream_budget=budget) as p:
        assert p.run(2) == 2  # a captured iteration of the plan that stays
        with refuse(name):
            with contextlib.suppress(L.LpaError):
                p.set_dispatch(L.Dispatch.FORCE, L.Variant.TWO_PASS)
            try:
                ch = p.iterate()
            except L.LpaError as e:  # no memory for the old lists either
                assert e.status == L.Status.OOM
            else:
                assert ch == changed[2] and np.array_equal(p.labels(), hist[2])
                p.set_labels(hist[1])
        _check(p, hist, changed, 2)
        assert p.run(3) == 3
        assert np.array_equal(p.labels(), hist[5])
        p.set_dispatch(L.Dispatch.FORCE, L.Variant.TWO_PASS)  # there is memory now
        p.init_labels()
        for it in range(3):
            _check(p, hist, changed, it)


def test_failed_tune(case):
    g, want = case
    hist, changed = want[0]
    with L.Propagator(g, dispatch=L.Dispatch.FORCE, force_variant=int(L.Variant.TWO_PASS)) as p:
        before = p.get_tune()
        with refuse("count items"):
            with pytest.raises(L.LpaError) as e:
                p.set_tune(1, 1, before.warp_max_degree, before.warp_claim)  # more items
            assert e.value.status == L.Status.OOM
        assert p.get_tune().as_tuple() == before.as_tuple()
        for it in range(3):
            _check(p, hist, changed, it)


def test_learner_without_memory(case):
    """Explorations that do not fit: the heuristic plan stays."""
    g, want = case
    hist, changed = want[CMS]
    with L.Propagator(g, cms_threshold=CMS, dispatch=L.Dispatch.LEARNED) as p:
        with refuse("two-pass scratch"):
            for it in range(6):
                _check(p, hist, changed, it)
        p.init_labels()
        p.run(6)
        assert np.array_equal(p.labels(), hist[5])


@pytest.mark.parametrize("cms", [0, CMS])
@pytest.mark.parametrize("thresh", [0, 16])
def test_hubs_without_scratch(case, thresh, cms):
    """No memory for the hubs' labels: blocks of k_iterate decode and count them."""
    g, want = case
    hist, changed = want[cms]
    row, clm = g.csr()
    g2 = L.HostGraph.from_csr(row, clm).compress(thresh, 128)
    with refuse("two-pass scratch"):
        p = L.Propagator(g2, cms_threshold=cms)
    with p:
        for it in range(3):
            _check(p, hist, changed, it)
        p.init_labels()
        p.run(6)
        assert np.array_equal(p.labels(), hist[5])


@pytest.mark.parametrize("gather", [0, 1, 2])
@pytest.mark.parametrize("stage", [0, 1, 2])
def test_without_records(case, stage, gather):
    """No memory for the segment records: decode groups cover the residual segments."""
    g, want = case
    hist, changed = want[CMS]
    with refuse("segment records"):
        p = L.Propagator(g, cms_threshold=CMS, dispatch=L.Dispatch.FORCE, force_variant=int(L.Variant.TWO_PASS))
    with p:
        p.set_tune(*p.get_tune().as_tuple()[:5], gather, stage)
        for it in range(3):
            _check(p, hist, changed, it)


def test_count_tables_only_where_used(case):
    """Exact hubs above the shared table run through the two-pass kernels: heavy
    items of the small CSR (degree 1024 to 2047) need no global tables for them."""
    g, want = case
    hist, changed = want[0]
    row, clm = g.csr()
    deg = np.diff(row)
    assert ((deg > 1023) & (deg < 2048)).any()
    with refuse("global count tables"):
        with L.Propagator(L.HostGraph.from_csr(row, clm).compress(2048, 2048)) as p:
            for it in range(3):
                _check(p, hist, changed, it)
            p.set_dispatch(L.Dispatch.FORCE, L.Variant.BLOCK)
            p.init_labels()
            p.run(6)
            assert np.array_equal(p.labels(), hist[5])
        small = L.HostGraph.from_csr(row, clm).compress(8192, 8192)  # the hubs in the small CSR
        with pytest.raises(L.LpaError) as e:
            L.Propagator(small)
        assert e.value.status == L.Status.OOM
    with L.Propagator(small) as p:
        for it in range(3):
            _check(p, hist, changed, it)


def test_refused_graph_leaves_no_memory():
    """A malformed stream is refused after the degree pass: all its memory comes back."""
    arr = L.HostGraph.road(1000, 1000, seed=3).compress(0, 128).arrays()
    mid = len(arr["words"]) // 2
    arr["words"][mid:mid + 8] = 0
    free = []
    for _ in range(6):  # 4 MB of interval counts and 4 MB of hub list each
        with pytest.raises(L.LpaError) as e:
            L.Propagator(L.desc_from_arrays(arr))
        assert e.value.status == L.Status.BAD_STREAM
        free.append(torch.cuda.mem_get_info(0)[0])
    assert free[0] - free[-1] < 4 << 20


def test_position_arrays_end_at_the_last_hub():
    """One hub, first in position order, among 200,000 compressed vertices: what the
    two-pass kernels keep by position (28 bytes each) does not cover them all."""
    n, d = 200000, 2000
    v = np.arange(n)
    lists = [np.arange(1, 1 + d)] + [np.array([x - 1]) for x in v[1:]]
    row = np.concatenate([[0], np.cumsum([len(x) for x in lists])]).astype(np.uint64)
    clm = np.concatenate(lists).astype(np.uint32)
    hist, changed = oracle.lp_run(row, clm, 3, 0, 1)
    g = L.HostGraph.from_csr(row, clm).compress(0, 128)
    with refuse("two-pass scratch"):
        with L.Propagator(g) as p:
            without = p.get_info().device_bytes
    for budget in (0, 1 << 20):
        with L.Propagator(g, stream_budget=budget) as p:
            if not budget:
                assert p.get_info().device_bytes - without < 1 << 20
            for it in range(3):
                _check(p, hist, changed, it)
            drow, dclm = p.decode_csr()  # of a streamed handle: needs every position's
            assert np.array_equal(drow, row) and np.array_equal(dclm, clm)
            p.set_dispatch(L.Dispatch.FORCE, L.Variant.TWO_PASS)
            p.init_labels()
            for it in range(3):
                _check(p, hist, changed, it)
