"""Rate-coded networks held on chip for a whole run (one persistent kernel on
a cluster or on one CTA per SM) against the engine of one launch per phase:
the same bits in double precision, rounding differences in single precision."""
import numpy as np
import pytest

import annarchy_b200 as ann
from annarchy_b200 import workloads as wl
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in,n,p_in,p_rec,ctas", [
    (3, 5, 0.6, 0.6, 148), (7, 33, 0.3, 0.3, 1), (1, 1, 1.0, 1.0, 1), (100, 400, 0.1, 0.05, None),
    (100, 400, 0.1, 0.05, 16), (50, 1501, 0.1, 0.05, 148), (1000, 4000, 0.1, 0.02, None)])
@pytest.mark.parametrize("precision", ["double", "float"])
def test_runs_match_the_oracle(n_in, n, p_in, p_rec, ctas, precision):
    rn = wl.rate_net(seed=4, n_in=n_in, n_out=n, p_in=p_in, p_rec=p_rec, steps=61)
    cfg = {"resident_ctas": ctas} if ctas else {}
    net, pop, mon = wl.build_rate_network(rn, precision, **cfg)
    net.compile()
    assert net.engine == "resident"
    for k in (1, 20, 40):
        net.simulate_steps(k)
    _, ref = orc.rate_run(rn, 61, trace=True)
    ref = np.asarray(ref).reshape(61, n)
    r, trace = np.asarray(pop.r), mon.get("r")
    if precision == "double":
        assert np.array_equal(trace, ref) and np.array_equal(r, ref[-1])
    else:
        # float32 sums of up to a few hundred terms, 61 contracting steps
        assert np.linalg.norm(trace - ref) <= 1e-5 * np.linalg.norm(ref)
        assert np.array_equal(r, trace[-1])
    net.close()


def _model(precision, engine, ctas=None, wdt=None):
    """Two populations with parameters of one name, two targets, views on
    both sides, an unconnected neuron range, a local parameter, recordings of
    a view, of a sum and of an input, and recorded periods."""
    net = ann.Network(dt=1.0, seed=1)
    net.config(precision=precision, engine=engine, **({"resident_ctas": ctas} if ctas else {}),
               **({"weight_dtype": wdt} if wdt else {}))
    rng = np.random.default_rng(2)
    inp = net.create(37, ann.Neuron(parameters="r = 0.0"))
    nrn = ann.Neuron(parameters="""
        tau = 10.0 : population
        gain = 1.0
    """, equations="""
        mp = gain * sum(exc) - sum(inh)
        tau * dr/dt + r = mp : min=0.0, max=2.0
    """)
    a, b = net.create(130, nrn), net.create(75, nrn)

    def w(pre, post, p, scale):
        m = wl.bernoulli_csr_skip(rng, post, pre, p, lambda k: rng.normal(0.0, scale, k))
        return wl.to_from_sparse(m)

    net.connect(inp, a, "exc").from_sparse(abs(w(37, 130, 0.4, 0.3)))
    net.connect(a[10:90], b[5:60], "exc").from_sparse(w(80, 55, 0.3, 0.2))
    net.connect(b, a, "inh").from_sparse(w(75, 130, 0.1, 0.2))
    net.connect(b, b, "exc").from_sparse(w(75, 75, 0.05, 0.2))
    ms = [net.monitor(a, ["r", "sum(exc)"], period=3.0), net.monitor(b[7:31], "mp"), net.monitor(inp, "r")]
    net.compile()
    a.gain = rng.uniform(0.5, 1.5, 130)
    return net, inp, a, b, ms


@pytest.mark.parametrize("precision,wdt", [("double", None), ("float", None), ("float", "bfloat16")])
@pytest.mark.parametrize("ctas", [2, 16, 148])
def test_forms_match_the_engine_of_launches(precision, wdt, ctas):
    out = []
    for engine in ("grid", "auto"):
        net, inp, a, b, ms = _model(precision, engine, ctas if engine == "auto" else None, wdt)
        assert net.engine == ("grid" if engine == "grid" else "resident")
        rng = np.random.default_rng(3)
        for k in (5, 1, 12):
            inp.r = rng.uniform(0.0, 1.0, 37)
            net.simulate_steps(k)
        net.projections[3].w = 0.25                     # weights set between runs
        ms[1].pause()
        net.simulate_steps(7)
        ms[1].resume()
        net.set_time(100.0)
        net.simulate_steps(9)
        res = [a.r, a.mp, a.sum("exc"), a.sum("inh"), b.r, b.mp, ms[0].get("r"), ms[0].get("sum(exc)"),
               ms[1].get("mp"), ms[2].get("r")]
        net.reset()
        net.simulate_steps(4)
        out.append([np.asarray(x) for x in res + [a.r, b.r]])
        net.close()
    for x, y in zip(*out):
        assert x.shape == y.shape
        if precision == "double":
            assert np.array_equal(x, y)
        else:
            assert np.linalg.norm(x - y) <= 1e-5 * np.linalg.norm(x)
