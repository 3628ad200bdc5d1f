"""Vertices at the edges of the kernels' degree limits, hubs on every path they
take (block variant, two-pass, hash shares), and whole runs in one launch."""
import numpy as np
import pytest

import lpa_b200 as L
import oracle

pytestmark = pytest.mark.gpu

N = 12000
DEGREES = [1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 127, 128, 129, 511, 512, 1023, 1024, 1025, 2047, 2048, 2049,
           4095, 4096, 4097, 6000, 8193, 11999]


def _slot_hash(x):
    """The device's table hash (common.cuh slot_hash)."""
    x = np.asarray(x, np.uint64) & 0xFFFFFFFF
    for s, m in ((16, 0x7FEB352D), (15, 0x846CA68B)):
        x ^= x >> np.uint64(s)
        x = (x * np.uint64(m)) & np.uint64(0xFFFFFFFF)
    return x ^ (x >> np.uint64(16))


def _edge_graph(seed):
    """N vertices; every degree of DEGREES several times, lists with and
    without runs of consecutive ids (short, long, the whole list)."""
    rng = np.random.default_rng(seed)
    deg = np.concatenate([np.repeat(DEGREES[:20], 40), np.repeat(DEGREES[20:], 3), rng.integers(0, 12, N)])[:N]
    rng.shuffle(deg)
    rows = []
    for v in range(N):
        d = int(deg[v])
        kind = v % 3
        if kind == 0 or d > N // 2:
            ids = rng.choice(N, d, replace=False)
        elif kind == 1:  # one run
            start = int(rng.integers(0, N - d + 1))
            ids = np.arange(start, start + d)
        else:  # half in short runs
            starts = rng.choice(N // 16, d // 8 + 1, replace=False) * 16
            runs = (starts[:, None] + np.arange(6)).ravel()
            ids = np.unique(np.concatenate([runs, rng.choice(N, d, replace=False)]))
            ids = rng.choice(ids, d, replace=False)
        rows.append(np.sort(ids).astype(np.uint32))
    row = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.uint64)
    return row, np.concatenate(rows)


@pytest.fixture(scope="module")
def edge():
    return _edge_graph(3)


@pytest.mark.parametrize("cms", [0, 700, 2049])
@pytest.mark.parametrize("thresh", [0, 16, 128])
@pytest.mark.parametrize("variant", [None, L.Variant.WARP, L.Variant.BLOCK, L.Variant.TWO_PASS],
                         ids=lambda v: "fixed" if v is None else v.name.lower())
def test_degree_limits(edge, variant, thresh, cms):
    row, clm = edge
    g = L.HostGraph.from_csr(row, clm).compress(thresh, 128)
    hist, changed = oracle.lp_run(row, clm, 4, cms, 1)
    opts = dict(cms_threshold=cms, cms_seed=1)
    if variant is not None:
        opts.update(dispatch=L.Dispatch.FORCE, force_variant=int(variant))
    with L.Propagator(g, **opts) as p:
        for it in range(4):
            assert p.iterate() == changed[it], f"iteration {it + 1}"
            assert np.array_equal(p.labels(), hist[it]), f"iteration {it + 1}"
        p.init_labels()
        assert p.run(4) == 4  # the captured loop
        assert np.array_equal(p.labels(), hist[3])
        # from the hubs' scratch to the whole one and back
        p.set_dispatch(L.Dispatch.FORCE, L.Variant.TWO_PASS)
        p.set_dispatch(L.Dispatch.FIXED)
        p.init_labels()
        assert p.iterate() == changed[0]
        assert np.array_equal(p.labels(), hist[0])


def test_encode_and_decode(edge):
    row, clm = edge
    host = L.HostGraph.from_csr(row, clm).compress(16, 128).arrays()
    g = L.HostGraph.from_csr(row, clm).compress(16, 128, device=0)
    dev = g.arrays()
    for k in ("words", "offsets", "vertices", "small_graph", "small_offset"):
        assert np.array_equal(host[k], dev[k]), k
    with L.Propagator(g) as p:
        drow, dclm = p.decode_csr()
    assert np.array_equal(drow, row)
    for v in range(N):
        a, b = int(row[v]), int(row[v + 1])
        assert np.array_equal(np.sort(dclm[a:b]), clm[a:b]), v


def test_hash_share_overfull():
    """All labels of a hub in one hash share: the share is counted in parts."""
    n, d = 20000, 5000
    cand = np.arange(1, 1 << 17, dtype=np.uint32)
    pick = cand[_slot_hash(cand) >> np.uint64(30) == 2]
    labels = np.resize(pick, n).astype(np.uint32)  # different for every neighbour
    rng = np.random.default_rng(0)
    ids = np.sort(rng.choice(np.arange(1, n), d, replace=False)).astype(np.uint32)
    labels[ids[77]] = labels[ids[4000]] = labels[ids[123]]  # the most frequent
    row = np.zeros(n + 1, np.uint64)
    row[1:] = d
    assert len(np.unique(labels[ids])) > 4096
    g = L.HostGraph.from_csr(row, ids).compress(0, 128)
    with L.Propagator(g, dispatch=L.Dispatch.FORCE, force_variant=int(L.Variant.TWO_PASS)) as p:
        p.set_labels(labels)
        p.iterate()
        want = labels.copy()
        want[0] = labels[ids[123]]
        assert np.array_equal(p.labels(), want)


def test_malformed_hub_is_refused(edge):
    """64 zero bits inside a hub's stream are no code: the degree pass says so."""
    row, clm = edge
    arr = L.HostGraph.from_csr(row, clm).compress(0, 128).arrays()
    deg = np.diff(row.astype(np.int64))[arr["vertices"]]
    p = int(np.flatnonzero((deg == 6000) & (arr["vertices"] % 3 != 1))[0])
    w = int((arr["offsets"][p] + arr["offsets"][p + 1]) // 64)
    arr["words"][w:w + 12] = 0
    with pytest.raises(L.LpaError) as e:
        L.Propagator(L.desc_from_arrays(arr))
    assert e.value.status == L.Status.BAD_STREAM


@pytest.mark.parametrize("width,height", [(2, 1), (3, 5), (31, 33), (64, 65), (200, 301)])
@pytest.mark.parametrize("early", [False, True])
def test_run_in_one_launch(width, height, early):
    """A road grid's plan is all k_packed: lpa_run's one launch against lpa_iterate."""
    g = L.HostGraph.road(width, height, seed=7)
    row, clm = g.csr()
    g.compress(0, 128)
    hist, changed = oracle.lp_run(row, clm, 25, 0, 1, early_exit=early)
    with L.Propagator(g) as p:
        for _ in range(2):  # an odd number of iterations swaps the buffers
            p.init_labels()
            done = p.run(25, early_exit=early)
            assert done == len(hist)
            assert np.array_equal(p.labels(), hist[-1])
            assert list(p.changed_history(done)) == changed
            p.run(3)
