"""Two populations of one neuron model with different parameter values on one
cluster (one weight per projection with and without delays, distributed
weights): the launch plan's spikes and states, bit for bit in double
precision. A parameter of one population does not hide a constant from the
other."""
import numpy as np
import pytest

import annarchy_b200 as ann
from annarchy_b200 import workloads as wl
from annarchy_b200.runtime import lib as L

FORMS = ["masks", "delays", "cluster"]


def _net(form, precision, engine, n_e=700, n_i=90):
    net = ann.Network(dt=0.1, seed=0)
    net.config(precision=precision, engine=engine)
    E = net.create(n_e, wl.coba_neuron(dict(wl.COBA_PARAMS, I=35.0)))
    I = net.create(n_i, wl.coba_neuron(dict(wl.COBA_PARAMS, I=33.0, tau=12.0, Vr=-58.0)))
    rng = np.random.default_rng(1)
    for k, (pre, post, target, p, w) in enumerate((
            (E, E, "exc", 0.05, 0.031), (E, I, "exc", 0.1, 0.023), (I, E, "inh", 0.1, 0.11), (I, I, "inh", 0.1, 0.07))):
        m = wl.bernoulli_csr_skip(rng, len(post), len(pre), min(p, 20.0 / len(pre)), w)
        if form == "cluster":
            m.data *= rng.uniform(0.5, 1.5, m.nnz)
        delay = (0.5, 0.0, 1.2, 0.3)[k] if form == "delays" else 0.0
        net.connect(pre, post, target).from_sparse(wl.to_from_sparse(m), delay)
    mons = net.monitor(E, "spike"), net.monitor(I, "spike")
    E.v = rng.uniform(-60.0, -50.0, n_e)
    I.v = rng.uniform(-58.0, -50.0, n_i)
    return net, E, I, mons


@pytest.mark.parametrize("precision", ["double", "float"])
@pytest.mark.parametrize("form", FORMS)
def test_modules_compile(form, precision):
    net, *_ = _net(form, precision, "auto")
    mod = net.generate_code()
    assert mod.kernels == ["anb_cluster_run"]
    size, log = L.nvrtc_compile(mod.source, mod.options)
    assert size > 0 and "error" not in log.lower()


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [(700, 90), (33, 130), (2049, 500)])
@pytest.mark.parametrize("form", FORMS)
def test_double_runs_match_the_launch_plan(form, sizes):
    out = []
    for engine in ("grid", "auto"):
        net, E, I, mons = _net(form, "double", engine, *sizes)
        net.compile()
        assert (net._backend.module.kernels == ["anb_cluster_run"]) == (engine == "auto")
        for k in (1, 30, 269):
            net.simulate_steps(k)
        out.append([x for m in mons for x in m.spike_arrays()] + [E.v, E.g_exc, E.g_inh, I.v, I.g_exc])
        net.close()
    assert out[0][0].size > sizes[0] // 4 and out[0][2].size > sizes[1] // 4
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("form", FORMS)
def test_float_runs_follow_double(form):
    out = []
    for precision in ("double", "float"):
        net, E, I, mons = _net(form, precision, "auto")
        net.compile()
        net.simulate_steps(20)
        out.append([E.v, I.v, E.g_exc, I.g_exc])
        net.close()
    for a, b in zip(*out):
        # 20 steps of at most 50 roundings each of values up to 64
        np.testing.assert_allclose(a, b, atol=20 * 50 * 2.0**-24 * 64)


@pytest.mark.gpu
@pytest.mark.parametrize("delay", [0.0, 0.5])
def test_a_parameter_hides_a_constant_in_its_population_only(delay):
    net = ann.Network(dt=1.0, seed=0)
    net.constant("gain", 3.0)
    eq = dict(equations="v = gain + g_exc", spike="v > 100.0", reset="v = 0.0")
    A = net.create(40, ann.Neuron(parameters="gain = 5.0 : population", **eq))
    B = net.create(40, ann.Neuron(**eq))
    net.connect(A, B, "exc").one_to_one(1.0, delays=delay)
    net.compile()
    assert net._backend.module.kernels == ["anb_cluster_run"]
    net.simulate_steps(2)
    assert np.all(A.v == 5.0) and np.all(B.v == 3.0)
    net.close()
