"""Batched instances in double precision with one weight per projection
(events counted per neuron and step): every instance bit for bit its oracle
run, from bursts of thousands of spikes (longer than the spike list) to
instances without a partner on their CTA; several weights keep the ordered
additions."""
import numpy as np
import pytest

from annarchy_b200 import workloads as wl
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _nets(sizes, burst, steps, spread):
    out = []
    for i, n in enumerate(sizes):
        cn = wl.coba_net(seed=30 + i, n=n, p=min(0.5, 30.0 / n), w_exc=0.3 + 0.05 * i, w_inh=1.5, drive=22.0,
                         steps=steps)
        if burst:
            cn.v0[:] = -60.0 + 10.0 * (np.arange(n) % burst) / burst
        if spread:
            for m in (cn.w_exc, cn.w_inh):
                m.data *= np.random.default_rng(i).uniform(0.5, 1.5, m.nnz)
        out.append(cn)
    return out


@pytest.mark.parametrize("sizes,burst,ctas,spread", [
    ([5, 33, 64], 1, 2, False), ([401, 37, 1000, 255], 2, 2, False), ([2049], 1, None, False),
    ([3000, 400, 1200], 3, 2, False), ([401, 37, 300], 0, 1, True)])
def test_instances_match_their_oracle(sizes, burst, ctas, spread):
    steps = 211
    cns = _nets(sizes, burst, steps, spread)
    refs = [orc.coba_run(cn, steps=steps, max_spikes=cn.n * steps) for cn in cns]
    b, members = wl.build_batch(cns, "double", **({"ctas": ctas} if ctas else {}))
    b.compile()
    assert b.counted == (not spread)
    for k in (1, 60, 150):
        b.simulate_steps(k)
    for (net, pop, mon), ref in zip(members, refs):
        s, i = mon.spike_arrays()
        assert np.array_equal(s, ref["spike_steps"]) and np.array_equal(i, ref["spike_idx"])
        for name in ("v", "g_exc", "g_inh"):
            assert np.array_equal(pop.get(name), ref[name]), name
    b.close()
