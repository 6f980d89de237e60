"""Compensated variables in single precision: a value that is set is the
value, without the rounding error carried for the former one; the errors last
from run to run."""
import numpy as np
import pytest

import annarchy_b200 as ann

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 1000])
def test_a_value_set_between_runs_is_exact(n):
    net = ann.Network(dt=0.1, seed=0)
    net.config(precision="float", engine="grid")
    pop = net.create(n, ann.Neuron(equations="7.0 * dx/dt = -x", spike="x > 100.0", reset="x = 0.0"))
    net.compile()
    pop.x = np.linspace(1.0, 3.0, n)
    net.simulate_steps(37)
    pop.x = 0.0
    net.simulate_steps(5)
    assert np.all(np.asarray(pop.x) == 0.0)
    net.close()


@pytest.mark.parametrize("steps", [1, 7])
def test_delayed_runs_in_pieces_round_like_one(steps):
    """With synaptic delays the carried errors of a small network last from
    run to run, as on the launch plan (no transmissions: the same bits)."""
    out = []
    for engine, k in (("grid", 420), ("auto", 420), ("auto", steps)):
        net = ann.Network(dt=0.1, seed=0)
        net.config(precision="float", engine=engine)
        pop = net.create(70, ann.Neuron(parameters="I = 0.0", equations="""
            7.0 * dx/dt = I - x + g_exc
            5.0 * dg_exc/dt = -g_exc
        """, spike="x > 100.0", reset="x = 0.0"))
        net.connect(pop, pop, "exc").one_to_one(0.5, delays=0.5)
        net.compile()
        assert (net._backend.masks is not None) == (engine == "auto")
        pop.I = np.linspace(1.0, 30.0, 70)
        for _ in range(420 // k):
            net.simulate_steps(k)
        out.append(np.asarray(pop.x))
        net.close()
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
