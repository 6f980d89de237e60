"""Models whose parameters or constants carry the names of a run's first step
and number of steps: the kernels that run many steps keep such names to
themselves."""
import numpy as np
import pytest

import annarchy_b200 as ann
from annarchy_b200 import workloads as wl
from annarchy_b200.runtime import lib as L

KINDS = ["rate", "masks", "delays", "cluster"]


def _net(kind, precision, engine, constant):
    """t0 and nsteps as the population's parameters or as constants."""
    net = ann.Network(dt=1.0 if kind == "rate" else 0.1, seed=0)
    net.config(precision=precision, engine=engine)
    extra = {"t0": 0.25, "nsteps": 0.5}
    if constant:
        for name, value in extra.items():
            net.constant(name, value)
    decl = "" if constant else "\n".join(f"{k} = {v} : population" for k, v in extra.items())
    if kind == "rate":
        pop = net.create(60, ann.Neuron(parameters="tau = 10.0 : population\n" + decl,
                                        equations="tau * dr/dt + r = t0 + nsteps * sum(exc)"))
    else:
        pop = net.create(60, ann.Neuron(parameters="tau = 20.0 : population\nVt = 1.0 : population\n" + decl, equations="""
            tau * dv/dt = 6.0 * t0 + nsteps * g_exc - v
            5.0 * dg_exc/dt = -g_exc
        """, spike="v > Vt", reset="v = 0.0"))
    rng = np.random.default_rng(1)
    w = wl.bernoulli_csr_skip(rng, 60, 60, 0.2, 0.1)
    if kind == "cluster":
        w.data *= rng.uniform(0.5, 1.5, w.nnz)
    net.connect(pop, pop, "exc").from_sparse(wl.to_from_sparse(w), 0.5 if kind == "delays" else 0.0)
    return net, pop


@pytest.mark.parametrize("constant", [False, True])
@pytest.mark.parametrize("precision", ["double", "float"])
@pytest.mark.parametrize("kind", KINDS)
def test_modules_compile(kind, precision, constant):
    net, pop = _net(kind, precision, "auto", constant)
    mod = net.generate_code()
    assert mod.kernels == ["anb_rate_run" if kind == "rate" else "anb_cluster_run"]
    size, log = L.nvrtc_compile(mod.source, mod.options)
    assert size > 0 and "error" not in log.lower()


@pytest.mark.gpu
@pytest.mark.parametrize("constant", [False, True])
@pytest.mark.parametrize("kind", KINDS)
def test_values_match_the_launch_plan(kind, constant):
    out = []
    for engine in ("grid", "auto"):
        net, pop = _net(kind, "double", engine, constant)
        net.compile()
        net.simulate_steps(300)
        out.append(np.asarray(pop.r if kind == "rate" else pop.v))
        net.close()
    assert out[0].max() > 0.1
    assert np.array_equal(*out)
