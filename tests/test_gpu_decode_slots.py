"""Spike rings of several instances decoded on the device by slot, step and
rank, against the host decoder slot by slot; more spikes than the pinned stage
holds, and long reads through the stage."""
import numpy as np
import pytest

from annarchy_b200.runtime import lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps,sizes,p", [(1, [1], 0.5), (40, [1, 7, 0, 33, 64], 0.03), (300, [40, 41], 0.05),
                                           (2000, [33, 100], 0.0), (700, [125] * 4, 0.2)])
def test_slots_match_the_host_decoder(steps, sizes, p):
    rng = np.random.default_rng(steps)
    words = sum(sizes)
    first = np.concatenate(([0], np.cumsum(sizes)))
    bits = (rng.random((steps, words * 32)) < p).astype(np.uint8)
    buf = np.packbits(bits, axis=1, bitorder="little").view(np.uint32).reshape(steps, words)
    nat = L.NativeNet(0)
    nat.initialize(0.1)
    nat.create("ring", buf)
    for t0 in (0, 10**10):                      # the second with a guess of the first's size
        s, r, off = nat.monitor_decode("ring", steps, words, words * 32, t0, slots=first)
        assert off[0] == 0 and off[-1] == s.size == r.size == int(bits.sum())
        for i in range(len(sizes)):
            hs, hr = L.bitmap_decode(np.ascontiguousarray(buf[:, first[i]:first[i + 1]]), 32 * sizes[i])
            assert np.array_equal(s[off[i]:off[i + 1]], hs + t0)
            assert np.array_equal(r[off[i]:off[i + 1]], hr)
    nat.close()


@pytest.mark.parametrize("n", [1, (1 << 18) - 1, 1 << 18, (1 << 18) + 1, (5 << 18) + 3])
def test_reads_around_the_stage_size(n):
    x = np.random.default_rng(n).integers(0, 2**32, n, dtype=np.uint32)
    nat = L.NativeNet(0)
    nat.initialize(0.1)
    nat.create("x", x)
    assert np.array_equal(nat.read("x"), x)
    assert np.array_equal(nat.read("x", count=n // 2, offset=n - n // 2), x[n - n // 2:])
    nat.close()
