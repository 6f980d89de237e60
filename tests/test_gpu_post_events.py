"""Post-spike events in the update kernels, from one bitmap word per CTA to a
full CTA, against a kernel of their own: the same weights, bit for bit, after
steps with few and with many spikes."""
import numpy as np
import pytest
import scipy.sparse as sp

import annarchy_b200 as ann
from annarchy_b200 import workloads as wl
from annarchy_b200.generator.codegen import CodeGenerator

pytestmark = pytest.mark.gpu


def _weights(n, fan, precision):
    net = ann.Network(dt=0.1, seed=4)
    net.config(precision=precision, engine="grid")
    A = net.create(n, ann.Neuron(parameters="p = 0.02 : population", equations="""
        x = Uniform(0.0, 1.0)
        5.0 * dg_exc/dt = -g_exc
    """, spike="x < p", reset="x = 1.0"))
    rng = np.random.default_rng(n)
    k = min(n, fan)
    m = sp.csr_matrix((rng.uniform(0.0, 0.5, n * k), np.concatenate([np.sort(rng.choice(n, k, replace=False)) for _ in range(n)]),
                       np.arange(0, n * k + 1, k)), shape=(n, n))
    p = net.connect(A, A, "exc", ann.STDP(**wl.STDP_PARAMS))
    p.from_sparse(wl.to_from_sparse(m))
    net.compile()
    kernels = net._backend.module.kernels
    net.simulate_steps(20)
    A.p = 0.4
    net.simulate_steps(5)
    A.p = 0.0
    net.simulate_steps(2)
    w = p.get("w", flat=True)
    net.close()
    return w, m.data, "proj0_post_event" in kernels


@pytest.mark.parametrize("precision", ["double", "float"])
@pytest.mark.parametrize("n,fan", [(1, 1), (31, 31), (33, 20), (257, 257), (1000, 256), (1000, 257), (4735, 300), (4737, 300),
                                   (9471, 30), (9473, 30), (20000, 20), (65535, 8)])
def test_weights_match_those_of_the_own_kernel(n, fan, precision, monkeypatch):
    w, w0, own = _weights(n, fan, precision)
    assert own == (precision == "float" and fan > 256 and 256 < n < 4736)
    monkeypatch.setattr(CodeGenerator, "post_fused", lambda self, proj: False)
    ref, _, own = _weights(n, fan, precision)
    assert own and np.array_equal(w, ref)
    assert n < 30 or not np.allclose(w, w0)
