"""Labels may take every 32-bit value: 0xFFFFFFFF has no key of its own in the
exact counters' tables, and wins or loses like any other."""
import numpy as np
import pytest

import lpa_b200 as L

pytestmark = pytest.mark.gpu

TOP = 0xFFFFFFFF


def _mode(labels):
    """Most frequent, the smallest on ties."""
    u, c = np.unique(labels, return_counts=True)
    return u[np.argmax(c)]


@pytest.mark.parametrize("thresh", [0, 8192])
@pytest.mark.parametrize("variant", [None, L.Variant.BLOCK, L.Variant.TWO_PASS],
                         ids=lambda v: "fixed" if v is None else v.name.lower())
@pytest.mark.parametrize("degree", [32, 700, 2100, 4000, 5000])
def test_top_label(degree, variant, thresh):
    """A hub with `top` labels 0xFFFFFFFF and `other` of a second label, the rest all different."""
    n = 6000
    rng = np.random.default_rng(degree)
    ids = np.sort(rng.choice(np.arange(1, n), degree, replace=False)).astype(np.uint32)
    row = np.zeros(n + 1, np.uint64)
    row[1:] = degree
    g = L.HostGraph.from_csr(row, ids).compress(thresh, max(thresh, 128))
    opts = {} if variant is None else dict(dispatch=L.Dispatch.FORCE, force_variant=int(variant))
    with L.Propagator(g, **opts) as p:
        for top, other in [(12, 8), (8, 12), (10, 10), (10, 9)]:
            labels = rng.permutation(np.arange(1, 1 << 20, dtype=np.uint32))[:n]
            at = rng.permutation(ids)
            labels[at[:top]] = TOP
            labels[at[top:top + other]] = 0xFFFFFFFE
            want = labels.copy()
            want[0] = _mode(labels[ids])
            p.set_labels(labels)
            p.iterate()
            assert np.array_equal(p.labels(), want), (top, other)
