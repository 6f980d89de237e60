"""Order of additions on the cluster with per-warp masks: two projections of
one target from disjoint bitmap words, several spikes per word and step, each
with its own weight; all of the first projection's events come before the
second's, as on the launch plan, bit for bit in double precision."""
import numpy as np
import pytest
import scipy.sparse as sp

import annarchy_b200 as ann
from annarchy_b200 import workloads as wl
from annarchy_b200.core.backend import CompiledNetwork
from annarchy_b200.generator.masks import Masks


def _net(engine, n, cut, delay, seed=3):
    net = ann.Network(dt=0.1, seed=0)
    net.config(precision="double", engine=engine)
    A = net.create(n, wl.coba_neuron(dict(wl.COBA_PARAMS, I=22.0)))
    rng = np.random.default_rng(seed)
    for lo, hi, target, w in ((0, cut, "exc", 0.31), (cut, n, "exc", 0.17), (0, cut, "inh", 0.6)):
        m = wl.bernoulli_csr_skip(rng, n, hi - lo, 0.3, w)
        net.connect(A[lo:hi], A, target).from_sparse(wl.to_from_sparse(sp.csr_matrix(m)), delay)
    mon = net.monitor(A, "spike")
    # groups of neurons with one potential spike together
    A.v = -60.0 + 10.0 * (np.arange(n) % 5) / 5
    return net, A, mon


@pytest.mark.parametrize("delay,tables", [(0.0, 2), (0.5, 2)])
def test_tables_hold_one_projection_of_a_target_without_delays(delay, tables):
    net, A, mon = _net("auto", 320, 160, delay)
    be = CompiledNetwork(net, dry=True)
    be.build()
    slots = Masks(be).slots()
    assert len(slots) >= tables
    if delay == 0.0:
        for s in slots:
            targets = [p.target for p, _, _ in s["projs"]]
            assert len(set(targets)) == len(targets)
    assert [p.id for s in slots for p, _, _ in s["projs"]] == [0, 1, 2]


@pytest.mark.gpu
@pytest.mark.parametrize("n,cut", [(64, 32), (320, 160), (1000, 512)])
@pytest.mark.parametrize("delay", [0.0, 0.5])
def test_projections_of_one_target_from_disjoint_words(n, cut, delay):
    out = []
    for engine in ("grid", "auto"):
        net, A, mon = _net(engine, n, cut, delay)
        net.compile()
        assert (net._backend.module.kernels == ["anb_cluster_run"]) == (engine == "auto")
        net.simulate_steps(150)
        out.append((*mon.spike_arrays(), A.v, A.g_exc, A.g_inh))
        net.close()
    assert out[0][0].size > n // 2
    for a, b in zip(*out):
        assert np.array_equal(a, b)
