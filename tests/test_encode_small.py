"""The GPU encoder on graphs with nothing or little to compress: the host encoder's arrays."""
import numpy as np
import pytest

import lpa_b200 as L

pytestmark = pytest.mark.gpu

GRAPHS = {
    "no_arcs": lambda: L.HostGraph.from_csr(np.zeros(8, np.uint64), np.zeros(0, np.uint32)),
    "one_vertex": lambda: L.HostGraph.from_csr(np.zeros(2, np.uint64), np.zeros(0, np.uint32)),
    "road": lambda: L.HostGraph.road(31, 29, seed=1),
    "road_900": lambda: L.HostGraph.road(900, 901, seed=1),
    "rmat": lambda: L.HostGraph.rmat(12, 16, seed=1),
    "copy": lambda: L.HostGraph.copy_model(30000, 30, seed=1),
}


@pytest.mark.parametrize("thresh", [0, 1, 4, 16, 100000])
@pytest.mark.parametrize("graph", GRAPHS)
def test_same_as_host(graph, thresh):
    g = GRAPHS[graph]()
    host = g.compress(thresh, max(thresh, 128)).arrays()
    host = {k: np.array(v) for k, v in host.items()}
    dev = g.compress(thresh, max(thresh, 128), device=0).arrays()
    assert host.keys() == dev.keys()
    for k in host:
        assert np.array_equal(host[k], dev[k]), k
