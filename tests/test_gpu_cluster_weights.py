"""Weights set after compile() on the cluster kernels act as on the launch
plan: a projection without synapses."""
import numpy as np
import pytest
import scipy.sparse as sp

import annarchy_b200 as ann
from annarchy_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["double", "float"])
@pytest.mark.parametrize("delay", [0.0, 0.5])
def test_weights_of_a_projection_without_synapses(delay, precision):
    net = ann.Network(dt=0.1, seed=0)
    net.config(precision=precision)
    A = net.create(70, wl.coba_neuron(dict(wl.COBA_PARAMS, I=30.0)))
    m = wl.bernoulli_csr_skip(np.random.default_rng(1), 70, 70, 0.2, 0.1)
    net.connect(A, A, "exc").from_sparse(wl.to_from_sparse(m), delay)
    none = net.connect(A, A, "inh")
    none.from_sparse(sp.lil_matrix((70, 70)), delay)
    net.compile()
    assert none.nb_synapses == 0 and net._backend.module.kernels == ["anb_cluster_run"]
    none.w = 0.5
    net.simulate_steps(20)
    assert np.all(A.g_inh == 0.0)
    net.close()
