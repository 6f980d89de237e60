"""Small spiking networks with one weight per projection on one cluster
(per-warp masks, spikes exchanged with asynchronous stores): the oracle's
raster and state bit for bit in double precision; other forms against the
grid engine."""
import numpy as np
import pytest

import annarchy_b200 as ann
from annarchy_b200 import workloads as wl
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,p,burst,size", [
    (5, 1.0, 1, None), (33, 0.5, 1, 2), (33, 0.5, 1, 1), (130, 0.3, 2, 4), (400, 0.1, 2, 1),
    (400, 0.1, 0, 16), (1000, 0.05, 3, None), (2049, 0.03, 0, None), (4000, 0.02, 2, None),
    (5000, 0.01, 30, None)])
def test_runs_match_the_oracle(n, p, burst, size):
    steps = 331
    cn = wl.coba_net(seed=6, n=n, p=p, w_exc=0.4, w_inh=1.5, drive=22.0, steps=steps, skip=True)
    if burst:                       # up to thousands of spikes in one step
        cn.v0[:] = -60.0 + 10.0 * (np.arange(n) % burst) / burst
    ref = orc.coba_run(cn, steps=steps, max_spikes=n * steps)
    net, P, mon = wl.build_coba_network(cn, "double", "local", **({"cluster_size": size} if size else {}))
    net.compile()
    assert "net__masks0" in net._backend.native.arrays
    for k in (1, 2, 100, 228):
        net.simulate_steps(k)
    s, i = mon.spike_arrays()
    assert np.array_equal(s, ref["spike_steps"]) and np.array_equal(i, ref["spike_idx"])
    for name in ("v", "g_exc", "g_inh"):
        assert np.array_equal(P.get(name), ref[name]), name
    net.close()


def _two(engine, precision):
    """Two populations of different sizes, projections with overlapping and
    descending pre-synaptic ranges onto one target, a silent projection."""
    net = ann.Network(dt=0.1, seed=0)
    net.config(precision=precision, engine=engine)
    params = dict(wl.COBA_PARAMS, I=22.0)
    # (parameters of one name in both populations share a value in the kernel's scope)
    A = net.create(700, wl.coba_neuron(params))
    rng = np.random.default_rng(1)

    def con(pre, post, target, p, w):
        m = wl.bernoulli_csr_skip(rng, len(post), len(pre), p, w)
        net.connect(pre, post, target).from_sparse(wl.to_from_sparse(m))

    con(A[0:320], A, "exc", 0.05, 0.31)
    con(A[200:500], A, "exc", 0.05, 0.17)
    con(A[0:200], A[100:300], "exc", 0.1, 0.23)
    con(A[500:700], A, "inh", 0.1, 1.1)
    con(A[320:500], A[3:9], "inh", 1e-9, 1.0)      # (no synapse)
    m = net.monitor(A, "spike")
    net.compile()
    A.v = rng.uniform(-60.0, -50.0, 700)
    return net, A, m


@pytest.mark.parametrize("precision", ["double", "float"])
def test_projections_of_one_target_keep_their_order(precision):
    out = []
    for engine in ("grid", "auto"):
        net, A, m = _two(engine, precision)
        net.simulate_steps(300)
        out.append((*m.spike_arrays(), A.v, A.g_exc, A.g_inh, A.get("g_inh")))
        net.close()
    assert out[0][0].size > 500
    for x, y in zip(*out):
        if precision == "double":
            assert np.array_equal(x, y)
        else:                       # float sums in another order: the same rates
            assert x.shape[0] > 0 and abs(x.astype(float).mean() - y.astype(float).mean()) <= 0.05 * abs(
                x.astype(float).mean())
