"""Double precision on the launch plan through steps with few and with very many
spikes: inboxes, walks of single rows, of a whole warp's rows and of all rows
give the bits of the kernels that walk every row each step, which a recorded
conductance selects. Rows of one length, long rows among short ones, groups of
neurons that reach the same targets; several projections per target; without
delays, with a uniform delay, with one delay per synapse, plastic."""
import numpy as np
import pytest
import scipy.sparse as sp

import annarchy_b200 as ann
from annarchy_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def _neuron():
    return ann.Neuron(parameters="p = 0.001 : population\ntau = 20.0 : population\nte = 5.0 : population", equations="""
        x = Uniform(0.0, 1.0)
        tau * dv/dt = -v + g_exc - g_inh
        te * dg_exc/dt = -g_exc
        te * dg_inh/dt = -g_inh
    """, spike="x < p", reset="v = 0.0")


def _matrix(rng, n_post, n_pre, fan, shape):
    """(post, pre) weights: `fan` synapses per row; "hubs": the rows 40..79 from
    every neuron; "groups": 100 successive rows from the same 60 neurons."""
    lens = np.minimum(rng.poisson(fan, n_post), n_pre)
    cols = [np.sort(rng.choice(n_pre, k, replace=False)) for k in lens]
    if shape == "hubs":
        cols[40:80] = [np.arange(n_pre)] * len(cols[40:80])
    if shape == "groups":
        for i in range(0, min(100, n_post)):
            cols[i] = np.arange(min(60, n_pre))
    ptr = np.concatenate([[0], np.cumsum([c.size for c in cols])])
    return sp.csr_matrix((rng.uniform(0.05, 0.15, ptr[-1]), np.concatenate(cols), ptr), shape=(n_post, n_pre))


def _run(n, fan, shape, kind, plan_rows, burst):
    net = ann.Network(dt=0.1, seed=4)
    net.config(precision="double", engine="grid")
    A = net.create(n, _neuron())
    rng = np.random.default_rng(n)
    cut = max(1, n // 3)
    projs = []
    for q, (pre, post, target) in enumerate(((A, A, "exc"), (A[:cut], A, "exc"), (A[cut:], A, "inh"))):
        m = _matrix(rng, len(post), len(pre), fan if q == 0 else fan / 4 + 1, shape)
        syn = ann.STDP(**wl.STDP_PARAMS) if kind == "plastic" and q == 0 else None
        d = {"none": None, "plastic": None, "uniform": 4, "synapse": rng.integers(1, 12, m.nnz)}[kind]
        p = net.connect(pre, post, target, syn)
        p.from_sparse(wl.to_from_sparse(m), wl.delay_arg(m, d, 0.1))
        projs.append(p)
    mon = net.monitor(A, "spike")
    if plan_rows:
        net.monitor(A, ["g_exc", "g_inh"])
    net.compile()
    assert bool(net._backend.inbox) != plan_rows
    for p, steps in ((0.001, 30), (burst, 25), (0.002, 30), (4 * burst, 3), (0.0, 20)):
        A.p = p
        net.simulate_steps(steps)
    out = [*mon.spike_arrays(), A.v, A.g_exc, A.g_inh]
    if kind == "plastic":
        out.append(projs[0].get("w", flat=True))
    net.close()
    return out


@pytest.mark.parametrize("kind", ["none", "uniform", "synapse", "plastic"])
@pytest.mark.parametrize("n,fan,shape,burst", [
    (5, 5, "even", 0.5), (33, 33, "even", 0.2), (300, 300, "even", 0.02), (1000, 400, "even", 0.04),
    (1000, 20, "hubs", 0.02), (1000, 6, "groups", 0.05), (4001, 60, "hubs", 0.01), (9000, 40, "groups", 0.05)])
def test_dense_and_sparse_steps_match_the_row_walk(n, fan, shape, burst, kind):
    a, b = (_run(n, fan, shape, kind, rows, burst) for rows in (False, True))
    assert np.bincount(a[0], minlength=108).max() >= min(n, 5)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


def test_dense_steps_with_two_neurons_per_thread():
    a, b = (_run(70001, 12, "groups", "none", rows, 0.1) for rows in (False, True))
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
