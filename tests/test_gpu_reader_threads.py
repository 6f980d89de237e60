"""Several threads read the arrays of one network, small ones and ones beyond
the pinned stage, while spikes are decoded: every thread gets its own."""
import threading

import numpy as np
import pytest

from annarchy_b200.runtime import lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1000, 1000), (1, 200_000, 30_000), (250_000, 270_000, 64, 4096)])
def test_threads_read_their_own_arrays(sizes):
    nat = L.NativeNet(0)
    nat.initialize(0.1)
    arrays = [np.random.default_rng(i).integers(0, 2**32, n, dtype=np.uint32) for i, n in enumerate(sizes)]
    for i, a in enumerate(arrays):
        nat.create(f"x{i}", a)
    ring = np.zeros((50, 4), dtype=np.uint32)
    ring[::5, 1] = 0x80000001
    nat.create("ring", ring)
    bad = []

    def read(i):
        for _ in range(400):
            if not np.array_equal(nat.read(f"x{i}"), arrays[i]):
                bad.append(i)
                return

    def decode():
        for _ in range(400):
            s, r = nat.monitor_decode("ring", 50, 4, 128)
            if s.tolist() != [x for x in range(0, 50, 5) for _ in (0, 1)] or r.tolist() != [32, 63] * 10:
                bad.append("spikes")
                return

    threads = [threading.Thread(target=read, args=(i,)) for i in range(len(sizes))] + [threading.Thread(target=decode)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    nat.close()
