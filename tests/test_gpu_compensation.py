"""Compensated variables in single precision: a value that is set is the
value, without the rounding error carried for the former one."""
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
