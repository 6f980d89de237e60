"""Synaptic delays on the cluster with per-warp masks (one weight per
projection): the oracle's raster and state bit for bit in double precision;
delays, weights and the time changed between runs against the grid engine's
plan."""
import numpy as np
import pytest

import annarchy_b200 as ann
from annarchy_b200 import workloads as wl
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _masked(net):
    return "net__masks0" in net._backend.native.arrays


@pytest.mark.parametrize("n,p,burst,size,d_exc,d_inh", [
    (5, 1.0, 1, None, 2, None), (33, 0.5, 1, 2, 3, (1, 9)), (130, 0.3, 2, 4, (1, 3), (2, 63)),
    (400, 0.1, 2, 1, 15, 8), (1000, 0.05, 3, None, (1, 21), None), (2049, 0.03, 0, None, None, 31),
    (3000, 0.02, 2, None, (1, 21), (1, 11)), (4000, 0.01, 30, None, 5, (4, 7))])
def test_delayed_runs_match_the_oracle(n, p, burst, size, d_exc, d_inh):
    steps = 331
    cn = wl.coba_net(seed=6, n=n, p=p, w_exc=0.4, w_inh=1.5, drive=22.0, steps=steps, skip=True)
    rng = np.random.default_rng(n)
    if burst:                       # up to thousands of spikes in one step
        cn.v0[:] = -60.0 + 10.0 * (np.arange(n) % burst) / burst
    delays = tuple(rng.integers(*d, m.nnz) if isinstance(d, tuple) else d
                   for d, m in ((d_exc, cn.w_exc), (d_inh, cn.w_inh)))
    ref = orc.coba_run(cn, orc.coba_projections(cn, delays=delays), steps=steps, max_spikes=n * steps)
    net, P, mon = wl.build_coba_network(cn, "double", "auto", delays=delays,
                                        **({"cluster_size": size} if size else {}))
    net.compile()
    assert net.engine == "grid" and _masked(net)
    for k in (1, 2, 7, 93, 228):    # (runs shorter than the delays, too)
        net.simulate_steps(k)
    s, i = mon.spike_arrays()
    assert np.array_equal(s, ref["spike_steps"]) and np.array_equal(i, ref["spike_idx"])
    for name in ("v", "g_exc", "g_inh"):
        assert np.array_equal(P.get(name), ref[name]), name
    net.close()


def _two(engine, precision):
    """Two populations of different history lengths; delayed, undelayed,
    per-synapse and overlapping projections onto one target."""
    net = ann.Network(dt=0.1, seed=0)
    net.config(precision=precision, engine=engine)
    params = dict(wl.COBA_PARAMS, I=22.0)
    A = net.create(700, wl.coba_neuron(params))
    B = net.create(90, wl.coba_neuron(params))
    rng = np.random.default_rng(1)
    out = []

    def con(pre, post, target, p, w, delays):
        m = wl.bernoulli_csr_skip(rng, len(post), len(pre), p, w)
        proj = net.connect(pre, post, target)
        proj.from_sparse(wl.to_from_sparse(m), delays=0.0 if delays is None else delays)
        out.append(proj)

    con(A[0:320], A, "exc", 0.05, 0.31, 1.2)
    con(A[200:500], A, "exc", 0.05, 0.17, None)
    con(A[0:200], A[100:300], "exc", 0.1, 0.23, 0.3)
    con(B, A, "exc", 0.1, 0.4, None)
    con(A[500:700], B, "inh", 0.1, 1.1, 0.7)
    con(B, B, "inh", 0.1, 0.2, None)
    out[4].delay = 0.5
    m = net.monitor(A, "spike")
    net.compile()
    A.v = rng.uniform(-60.0, -50.0, 700)
    B.v = rng.uniform(-60.0, -50.0, 90)
    return net, A, B, m, out


def _drive(engine, precision):
    net, A, B, m, projs = _two(engine, precision)
    used = [_masked(net)]
    net.simulate_steps(150)
    projs[0].delay = 0.4                   # events on their way follow the new delay
    net.simulate_steps(3)
    projs[0].delay = 1.0
    net.simulate_steps(60)
    projs[1].w = 0.21                      # one weight again
    net.simulate_steps(60)
    with pytest.raises(ValueError):
        projs[0].delay = 9.0
    w = np.full(projs[0].nb_synapses, 0.3)
    w[::2] = 0.25                          # no longer one weight
    projs[0].w = [x for x in np.split(w, np.cumsum(projs[0].dendrite_sizes())[:-1])]
    net.simulate_steps(90)
    out = (*m.spike_arrays(), A.v, A.g_exc, B.v, B.get("g_inh"))
    net.close()
    return used, out


def test_changes_between_runs_match_the_plan():
    used_a, a = _drive("auto", "double")
    used_g, g = _drive("grid", "double")
    assert used_a == [True] and used_g == [False]
    assert a[0].size > 500
    for x, y in zip(a, g):
        assert np.array_equal(x, y)


def test_changes_between_runs_float():
    _, a = _drive("auto", "float")
    _, g = _drive("grid", "float")
    # float sums in another order: the same spikes early on, the same rates
    early = min(100, int(a[0].max()))
    n = int((a[0] < early).sum())
    assert np.array_equal(a[0][:n], g[0][:n]) and np.array_equal(a[1][:n], g[1][:n])
    assert abs(a[0].size - g[0].size) <= 0.05 * g[0].size


@pytest.mark.parametrize("precision", ["double", "float"])
def test_a_new_time_and_cleared_spikes(precision):
    """What is on its way after the time is set, and after the population is
    cleared, is what the bitmaps (and lists) of the plan say."""
    out = []
    for engine in ("auto", "grid"):
        net, A, B, m, projs = _two(engine, precision)
        net.simulate_steps(40)
        net.set_current_step(1003)
        net.simulate_steps(1)
        x = [A.g_exc, B.get("g_inh")]
        net.reset()
        net.simulate_steps(2)
        out.append(x + [A.g_exc, A.v, B.v])
        net.close()
    for x, y in zip(*out):
        if precision == "double":
            assert np.array_equal(x, y)
        else:                              # sums of at most 64 float weights in another order
            np.testing.assert_allclose(x, y, rtol=64 * 2.0**-24, atol=1e-7)


def test_long_delays_and_explicit_engines():
    """Histories beyond shared memory stay on the plan; engine="local" still
    refuses delays, engine="grid" is the plan."""
    def make(engine, delay):
        cn = wl.coba_net(seed=2, n=400, p=0.05, steps=50)
        return wl.build_coba_network(cn, "double", engine, delays=(delay, None))[0]

    net = make("auto", 20000)
    net.compile()
    assert not _masked(net)
    net.simulate_steps(40)
    net.close()
    net = make("grid", 20)
    net.compile()
    assert not _masked(net)
    net.close()
    net = make("local", 20)
    with pytest.raises(NotImplementedError):
        net.compile()
    net.close()
