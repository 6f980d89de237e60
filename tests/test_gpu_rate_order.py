"""CSR projections in the launch of a panelled one (single precision): the sums
of a target have one order of additions, so that runs repeat bit for bit where
every row lies in at most two pieces of the panelled projection; and the values
are those of separate launches in the projections' order."""
import numpy as np
import pytest
import scipy.sparse as sp

import annarchy_b200 as ann
from annarchy_b200 import workloads as wl
from annarchy_b200.generator.codegen import CodeGenerator


def _rows(rng, n_post, n_pre, k):
    cols = np.sort(rng.integers(0, n_pre, (n_post, k)), axis=1)
    m = sp.csr_matrix((rng.normal(0.0, 1.0, n_post * k), cols.ravel(), np.arange(0, n_post * k + 1, k)), shape=(n_post, n_pre))
    m.sum_duplicates()
    return m


def _sums(n, n_in, targets, reps):
    """One panel of 9000 neurons on few CTAs: a row is one piece, or two where a
    warp's range ends."""
    rng = np.random.default_rng(n)
    mats = [_rows(rng, n, 9000, 20)] + [_rows(rng, n, n_in, 3) for _ in targets]
    net = ann.Network(dt=1.0, seed=0)
    net.config(precision="float", engine="grid", weight_dtype="float32", pcsr_ctas=max(4, n // 1700))
    A = net.create(n_in, ann.Neuron(parameters="r = 0.0"))
    B = net.create(n, ann.Neuron(equations="x = sum(exc) + 2.0 * sum(inh)\nr = r"))
    C = net.create(9000, ann.Neuron(parameters="r = 0.0"))
    net.connect(C, B, "exc").from_sparse(wl.to_from_sparse(mats[0]), storage_format="pcsr")
    for t, m in zip(targets, mats[1:]):
        net.connect(A, B, t).from_sparse(wl.to_from_sparse(m), storage_format="csr")
    A.r, C.r = rng.uniform(0.0, 1.0, n_in), rng.uniform(0.0, 1.0, 9000)
    net.compile()
    plan = len(net._backend.module.plan)
    out = []
    for _ in range(reps):
        net.simulate_steps(1)
        out.append(np.stack([B.x, B.sum("exc")]))
    net.close()
    return plan, out


def test_partners_do_not_add_to_shared_sums():
    """The launch's CTAs add the panelled projection's pieces to the target's sums
    in no fixed order; a CSR projection of the same target stays out of them."""
    net = ann.Network(dt=1.0, seed=0)
    net.config(precision="float", engine="grid")
    A = net.create(50, ann.Neuron(parameters="r = 0.0"))
    B = net.create(70, ann.Neuron(equations="r = sum(exc) + sum(inh)"))
    rng = np.random.default_rng(0)
    net.connect(A, B, "exc").from_sparse(wl.to_from_sparse(_rows(rng, 70, 50, 20)), storage_format="pcsr")
    for t in ("exc", "inh", "exc"):
        net.connect(A, B, t).from_sparse(wl.to_from_sparse(_rows(rng, 70, 50, 2)), storage_format="csr")
    source = net.generate_code().source
    sums = [line.rsplit(", ", 1)[1] for line in source.split("\n") if "__post_rank, " in line]
    assert sums == ["anb_p_proj1__ps);", "anb_p_pop1___sum_inh);", "anb_p_proj3__ps);"]


@pytest.mark.gpu
@pytest.mark.parametrize("n,n_in,targets", [(5000, 800, ["exc"]), (5000, 800, ["exc", "exc"]), (5000, 800, ["inh", "inh"]),
                                            (70001, 900, ["exc", "inh", "exc"])])
def test_partner_sums_have_one_order(n, n_in, targets, monkeypatch):
    plan, out = _sums(n, n_in, targets, 60)
    assert plan == 2
    for x in out[1:]:
        assert np.array_equal(x, out[0])
    monkeypatch.setattr(CodeGenerator, "rate_partners", lambda self: {})
    plan, ref = _sums(n, n_in, targets, 1)
    assert plan == 2 + len(targets)
    assert np.array_equal(ref[0], out[0])
