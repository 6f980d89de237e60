"""Single-precision sums of the resident engine are no further from 64 bits than
the launch plan's."""
import numpy as np
import pytest
import scipy.sparse as sp

import annarchy_b200 as ann
from annarchy_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def _errors(engine, m, x, **cfg):
    n = x.size
    net = ann.Network(dt=1.0, seed=0)
    net.config(precision="float", engine=engine, weight_dtype="float32", **cfg)
    A = net.create(n, ann.Neuron(parameters="r = 0.0"))
    B = net.create(n, ann.Neuron(equations="r = sum(exc)"))
    net.connect(A, B, "exc").from_sparse(wl.to_from_sparse(m), storage_format="csr")
    net.compile()
    assert net.engine == ("resident" if engine == "auto" else "grid")
    out = []
    for v in x.T if x.ndim > 1 else [x]:
        A.r = v
        net.simulate_steps(1)
        out.append((np.asarray(B.r) - m @ v) / (abs(m) @ v))
    net.close()
    return np.sqrt(np.mean(np.square(out)))


@pytest.mark.parametrize("n,fan,heavy", [(1000, 8, 0), (2000, 20, 0), (2000, 20, 50), (3000, 60, 0), (4000, 150, 5)])
def test_rows_round_no_worse_than_on_the_plan(n, fan, heavy):
    rng = np.random.default_rng(n + fan)
    lens = np.full(n, fan)
    lens[:heavy] = n
    cols = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in lens])
    w = rng.normal(0.0, 1.0, cols.size).astype(np.float32).astype(np.float64)
    m = sp.csr_matrix((w, cols, np.concatenate([[0], np.cumsum(lens)])), shape=(n, n))
    x = rng.random(n).astype(np.float32).astype(np.float64)
    # (thousands of rows: the ratio of two equal errors scatters by 2 %)
    assert _errors("auto", m, x) <= 1.04 * _errors("grid", m, x)
