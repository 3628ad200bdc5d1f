"""The GPU encoder works on its caller's thread."""
import os
import threading

import pytest

import lpa_b200 as L

pytestmark = pytest.mark.gpu


def test_no_threads_of_its_own():
    g = L.HostGraph.rmat(19, 16, seed=4)
    g.compress(16, 128, device=0)  # the CUDA runtime's own threads start here
    stop, most = threading.Event(), [0]

    def watch():
        while not stop.is_set():
            most[0] = max(most[0], len(os.listdir("/proc/self/task")))

    t = threading.Thread(target=watch)
    t.start()
    before = len(os.listdir("/proc/self/task"))
    for _ in range(4):
        g.compress(16, 128, device=0)
    stop.set()
    t.join()
    assert most[0] <= before
