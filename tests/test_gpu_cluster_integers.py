"""Whole-number variables of spiking neurons beyond 2**24 in single precision
on the cluster kernels: counted exactly, as on the launch plan."""
import numpy as np
import pytest

import annarchy_b200 as ann
from annarchy_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["masks", "delays", "lists", "grid"])
def test_counters_stay_whole(form):
    net = ann.Network(dt=0.1, seed=0)
    net.config(precision="float", engine="grid" if form == "grid" else "auto")
    pop = net.create(70, ann.Neuron(equations="""
        k = k + 1 : int
        5.0 * dg_exc/dt = -g_exc
        x = g_exc
    """, spike="x > 100.0", reset="x = 0.0"))
    rng = np.random.default_rng(1)
    w = wl.bernoulli_csr_skip(rng, 70, 70, 0.2, 0.1)
    if form == "lists":
        w.data *= rng.uniform(0.5, 1.5, w.nnz)
    net.connect(pop, pop, "exc").from_sparse(wl.to_from_sparse(w), 0.5 if form == "delays" else 0.0)
    net.compile()
    assert (net._backend.masks is not None) == (form in ("masks", "delays"))
    start = 2**24 + np.arange(70)
    pop.k = start
    net.simulate_steps(5)
    net.simulate_steps(6)
    assert np.array_equal(pop.k, start + 11)
    net.close()
