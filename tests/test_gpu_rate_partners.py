"""CSR projections summed by the launch of a panelled projection (single
precision, launch plan) against each projection's own launch and against
64-bit sums: rows of 0 to 300 synapses, several panels, views, one and two
partners, a target of their own."""
import numpy as np
import pytest
import scipy.sparse as sp

import annarchy_b200 as ann
from annarchy_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def _matrix(rng, n_post, n_pre, mean):
    lens = np.minimum(rng.poisson(mean, n_post), n_pre)
    lens[::7] = 0
    cols = [np.sort(rng.choice(n_pre, k, replace=False)) for k in lens]
    m = sp.csr_matrix((rng.normal(0.0, 1.0, int(lens.sum())), np.concatenate(cols).astype(np.int64) if lens.sum()
                       else np.zeros(0, np.int64), np.concatenate([[0], np.cumsum(lens)])), shape=(n_post, n_pre))
    return m


@pytest.mark.parametrize("n,n_in,fan,partners,target", [
    (33, 5, 20, 1, "exc"), (1000, 300, 60, 1, "exc"), (5001, 700, 40, 2, "exc"), (5001, 700, 40, 2, "inh"),
    (20011, 1000, 50, 1, "exc")])
def test_partners_match_their_own_launches(n, n_in, fan, partners, target):
    rng = np.random.default_rng(n)
    r_in, r0 = rng.uniform(0.0, 1.0, n_in), rng.uniform(0.0, 1.0, n)
    mats = [_matrix(rng, n, n, fan)] + [_matrix(rng, n - 2 * i, n_in, fan / 6) for i in range(partners)]
    out = []
    for big in ("pcsr", "csr"):
        net = ann.Network(dt=1.0, seed=0)
        net.config(precision="float", engine="grid", weight_dtype="float32")
        A = net.create(n_in, ann.Neuron(parameters="r = 0.0"))
        B = net.create(n, ann.Neuron(equations="x = sum(exc) + 2.0 * sum(inh)\nr = r"))
        for i, m in enumerate(mats[1:]):
            net.connect(A, B[i:n - i], target).from_sparse(wl.to_from_sparse(m), storage_format="csr")
        net.connect(B, B, "exc").from_sparse(wl.to_from_sparse(mats[0]), storage_format=big)
        A.r, B.r = r_in, r0
        net.compile()
        assert len(net._backend.module.plan) == (2 if big == "pcsr" else 2 + partners)
        steps = []
        for _ in range(3):
            net.simulate_steps(1)
            steps.append(np.asarray(B.x, dtype=np.float64))
        out.append(steps)
        net.close()
    f = np.float32
    want, scale = np.zeros(n), np.zeros(n)
    terms = [(mats[0], r0, 1.0, 0)] + [(m, r_in, 2.0 if target == "inh" else 1.0, i) for i, m in enumerate(mats[1:])]
    for m, r, factor, i in terms:
        m32 = m.astype(f).astype(np.float64)
        want[i:n - i] += factor * (m32 @ r.astype(f).astype(np.float64))
        scale[i:n - i] += factor * (abs(m32) @ r.astype(f).astype(np.float64))
    # every product and each of the at most `terms` additions rounds once
    bound = (max(int(np.diff(m.indptr).max()) for m in mats) + 8) * 2.0**-24 * len(terms) * scale + 1e-30
    for steps in out:
        for x in steps:
            assert np.all(np.abs(x - want) <= bound)
