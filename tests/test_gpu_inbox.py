"""Event-driven transmission in the reference's order on the grid engine in
double precision: one, a few and more events per post neuron and step than
its inbox holds, without delays, with a uniform delay and with one delay per
synapse, static and plastic, one and several neurons per thread, partial
bitmap words; and a delay changed, the time set and spikes cleared in mid-run.
The oracle gives the raster and the state bit for bit (plastic weights within
1e-12: the device's exponential)."""
import numpy as np
import pytest

from annarchy_b200 import workloads as wl
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _net(n, p, burst, steps, seed=5):
    cn = wl.coba_net(seed=seed, n=n, p=p, w_exc=0.4, w_inh=1.5, drive=22.0, steps=steps, skip=True)
    if burst:
        # groups of neurons with one potential spike together
        cn.v0[:] = -60.0 + 10.0 * (np.arange(n) % burst) / burst
    rng = np.random.default_rng(seed + 1)
    for m in (cn.w_exc, cn.w_inh):       # distinct weights: the order of additions shows
        m.data *= rng.uniform(0.5, 1.5, m.nnz)
    return cn


def _delays(kind, cn, rng):
    if kind == "uniform":
        return 7, 3
    if kind == "synapse":
        return rng.integers(1, 24, cn.w_exc.nnz), rng.integers(1, 24, cn.w_inh.nnz)
    return None, None


@pytest.mark.parametrize("n,p,burst,kind,steps", [
    (5, 1.0, 1, "none", 300), (33, 0.5, 1, "none", 400), (333, 0.2, 3, "none", 400),
    (333, 0.2, 3, "uniform", 400), (333, 0.2, 3, "synapse", 400), (1000, 0.05, 0, "synapse", 400),
    (4001, 0.02, 40, "none", 300), (70001, 0.0005, 200, "none", 150), (70001, 0.0005, 20, "uniform", 150),
    (270001, 0.0001, 40, "none", 120)])
def test_static_events_match_the_oracle(n, p, burst, kind, steps):
    cn = _net(n, p, burst, steps)
    d = _delays(kind, cn, np.random.default_rng(9))
    ref = orc.coba_run(cn, orc.coba_projections(cn, delays=d), steps=steps)
    net, P, mon = wl.build_coba_network(cn, "double", "grid", delays=d)
    net.compile()
    net.simulate_steps(steps)
    s, i = mon.spike_arrays()
    assert np.array_equal(s, ref["spike_steps"]) and np.array_equal(i, ref["spike_idx"])
    for name in ("v", "g_exc", "g_inh"):
        assert np.array_equal(P.get(name), ref[name]), name
    net.close()


@pytest.mark.parametrize("n,p,burst,steps", [(34, 0.6, 2, 400), (500, 0.1, 5, 400), (4001, 0.02, 0, 400)])
def test_plastic_events_match_the_oracle(n, p, burst, steps):
    cn = _net(n, p, burst, steps)
    w_ee = wl.stdp_matrix(cn, 4, p)
    projs = orc.coba_projections(cn, stdp_w_ee=w_ee, stdp=wl.STDP_PARAMS)
    ref = orc.coba_run(cn, projs, steps=steps)
    net, P, mon = wl.build_coba_network(cn, "double", "grid", stdp_w_ee=w_ee)
    net.compile()
    net.simulate_steps(steps)
    s, i = mon.spike_arrays()
    assert np.array_equal(s, ref["spike_steps"]) and np.array_equal(i, ref["spike_idx"])
    w = net.projections[0].get("w", flat=True)
    assert np.linalg.norm(w - projs[0].w) <= 1e-12 * np.linalg.norm(projs[0].w)
    assert np.linalg.norm(P.v - ref["v"]) <= 1e-12 * np.linalg.norm(ref["v"])
    net.close()


def test_delay_time_and_spikes_changed_between_runs():
    """Spikes in flight follow the bitmaps of the history ring: a delay set,
    the time set and the bitmaps cleared in mid-run act as with the kernels
    that walk every row, which a recorded conductance selects."""
    cn = _net(400, 0.1, 8, 160)
    out = []
    for record in (False, True):
        net, P, mon = wl.build_coba_network(cn, "double", "grid", delays=(9, 4))
        if record:
            net.monitor(P, ["g_exc", "g_inh"])
        net.compile()
        assert bool(net._backend.inbox) != record
        net.simulate_steps(40)
        net.projections[0].delay = 0.5
        net.simulate_steps(40)
        net.set_current_step(3)
        net.simulate_steps(40)
        net._backend.native.zero("pop0__spk")
        net.simulate_steps(40)
        out.append((*mon.spike_arrays(), P.v, P.g_exc, P.g_inh))
        net.close()
    assert out[0][0].size > 100
    for a, b in zip(*out):
        assert np.array_equal(a, b)
