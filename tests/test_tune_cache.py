"""The autotuner's cache: a result counts for the kernels it was measured with."""
import pytest

import lpa_b200 as L

pytestmark = pytest.mark.gpu


def test_results_of_other_kernels_do_not_count(tmp_path):
    g = L.HostGraph.rmat(12, 16, seed=2).compress(16, 128)
    opts = dict(cms_threshold=256, dispatch=L.Dispatch.FORCE, force_variant=int(L.Variant.TWO_PASS))
    cache = tmp_path / "tune.txt"
    with L.Propagator(g, **opts) as p:
        found = p.autotune(cache, repeats=1).as_tuple()
    line = cache.read_text()
    old = "v5|" + line.split(" ")[0].split("|", 1)[1]  # the key before segment records and hash shares
    cache.write_text(f"{old} 7 3 63 5 1 2 2 0.001\n")
    with L.Propagator(g, **opts) as p:
        p.autotune(cache, repeats=1)
    assert len(cache.read_text().splitlines()) == 2  # searched, and its result added
    cache.write_text(line)
    with L.Propagator(g, **opts) as p:
        assert p.autotune(cache, repeats=1).as_tuple() == found
    assert cache.read_text() == line
