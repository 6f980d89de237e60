"""Weights set after compile() on the cluster kernels act as on the launch
plan: one weight per projection and distributed ones, in either order, and a
projection without synapses."""
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


def _net(form, precision, engine, n=700):
    net = ann.Network(dt=0.1, seed=0)
    net.config(precision=precision, engine=engine)
    A = net.create(n, wl.coba_neuron(dict(wl.COBA_PARAMS, I=35.0)))
    rng = np.random.default_rng(1)
    projs = []
    for lo, hi, target, w in ((0, 400, "exc", 0.31), (400, n, "inh", 0.6), (100, 300, "exc", 0.2)):
        m = wl.bernoulli_csr_skip(rng, n, hi - lo, 0.03, w)
        if form == "many":
            m.data *= rng.uniform(0.5, 1.5, m.nnz)
        elif form == "table":
            m.data *= rng.choice([0.5, 0.75, 1.25], m.nnz)
        p = net.connect(A[lo:hi], A, target)
        p.from_sparse(wl.to_from_sparse(m))
        projs.append(p)
    mon = net.monitor(A, "spike")
    A.v = rng.uniform(-60.0, -50.0, n)
    return net, A, mon, projs


def _values(p, kind):
    rng = np.random.default_rng(7)
    n = p.nb_synapses
    w = {"one": np.full(n, 0.17), "few": rng.choice([0.1, 0.2], n), "more": 0.1 + 0.001 * rng.integers(0, 200, n),
         "many": rng.uniform(0.05, 0.4, n)}[kind]
    return list(np.split(w, np.cumsum(p.dendrite_sizes())[:-1]))


@pytest.mark.parametrize("precision", ["double", "float"])
@pytest.mark.parametrize("form,kinds", [
    ("one", ["one"]), ("one", ["one", "few", "one"]), ("one", ["many", "more"]), ("table", ["few", "one"]),
    ("table", ["more", "many", "few"]), ("many", ["one", "many"])])
def test_weights_set_between_runs(form, kinds, precision):
    out = []
    for engine in ("grid", "auto"):
        net, A, mon, projs = _net(form, precision, engine)
        net.compile()
        assert net.engine == ("grid" if engine == "grid" else "cluster")
        res = []
        net.simulate_steps(60)
        for i, kind in enumerate(kinds):
            p = projs[i % 3]
            p.w = _values(p, kind)
            if precision == "double":
                net.simulate_steps(70)
                res += [A.v, A.g_exc, A.g_inh]
            else:
                # the same state on both sides, then few steps: sums of up to 64
                # float32 weights in another order
                A.g_exc, A.g_inh, A.v = 0.0, 0.0, -60.0 + 11.0 * (37 * np.arange(700) % 700) / 700
                net.simulate_steps(3)
                res += [A.g_exc, A.g_inh]
        if precision == "double":
            res += list(mon.spike_arrays())
        out.append([np.asarray(x) for x in res])
        net.close()
    for x, y in zip(*out):
        if precision == "double":
            assert np.array_equal(x, y)
        else:
            assert x.max() > 0.0
            np.testing.assert_allclose(x, y, rtol=3 * 64 * 2.0**-24, atol=1e-7)


def _dense(engine, weights):
    net = ann.Network(dt=0.1, seed=0)
    net.config(precision="double", engine=engine)
    A = net.create(2000, wl.coba_neuron(dict(wl.COBA_PARAMS, I=35.0)))
    rng = np.random.default_rng(2)
    m = wl.bernoulli_csr_skip(rng, 2000, 2000, 0.5, 0.002)
    if weights:
        m.data *= rng.uniform(0.5, 1.5, m.nnz)
    p = net.connect(A, A, "exc")
    p.from_sparse(wl.to_from_sparse(m))
    A.v = rng.uniform(-60.0, -50.0, 2000)
    net.compile()
    return net, A, p, m


@pytest.mark.parametrize("weights", [False, True])
def test_lists_that_fit_no_cluster(weights):
    """One weight: the mask kernel, and the plan when the weights become
    different; different weights from the start: the plan, unless the cluster
    was asked for."""
    out = []
    for engine in ("grid", "auto"):
        net, A, p, m = _dense(engine, weights)
        assert net.engine == ("cluster" if engine == "auto" and not weights else "grid")
        net.simulate_steps(40)
        p.w = list(np.split(np.random.default_rng(5).uniform(0.001, 0.003, m.nnz), np.cumsum(p.dendrite_sizes())[:-1]))
        assert net.engine == "grid"
        net.simulate_steps(60)
        out.append([A.v, A.g_exc])
        net.close()
    assert out[0][1].max() > 0.0
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    if weights:
        with pytest.raises(RuntimeError):
            _dense("local", True)
