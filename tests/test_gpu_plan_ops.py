"""Operations of a step plan that C programs can add (include/annarchy_b200.h):
the block product that packs its rates every step, and kernels that run side by
side between two others."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

from annarchy_b200.core.backend import from_bf16, to_bf16
from annarchy_b200.generator.formats import bsr_arrays
from annarchy_b200.runtime import lib as L
from annarchy_b200.spmm import TILE, canonical_tiles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_post,n_pre,batch", [(1, 1, 16), (64, 64, 64), (200, 130, 128), (1000, 321, 32)])
def test_block_product_of_a_plan(n_post, n_pre, batch):
    rng = np.random.default_rng(n_post)
    w = sp.random(n_post, n_pre, 0.2, "csr", random_state=1, data_rvs=lambda k: rng.normal(0.0, 1.0, k))
    d = bsr_arrays(np.arange(n_post), w.indptr, w.indices, w.data, n_pre, TILE)
    vals = d["values"].reshape(-1, TILE, TILE).transpose(0, 2, 1)
    x = rng.uniform(0.0, 1.0, (batch, n_pre)).astype(np.float32)
    nat = L.NativeNet(0)
    nat.initialize(1.0)
    nat.create("p__brow", d["block_row_ptr"].astype(np.int32))
    nat.create("p__bcol", d["block_col"].astype(np.int32))
    nat.create("p__tiles", to_bf16(canonical_tiles(vals)))
    nat.create_empty("p__xt", np.uint16, (-(-n_pre // TILE) * batch * TILE,))
    nat.create("x", x)
    nat.create("y", np.zeros((batch, n_post), np.float32))
    nat.load_module('extern "C" __global__ void none() {}', [])
    nat.plan([])
    L.check("anb_plan_add_bsr_tc", nat.lib.anb_plan_add_bsr_tc(
        nat.h, b"p", b"x", b"y", int(d["n_block_rows"]), batch, n_pre, n_post, 0))
    nat.run(2)
    nat.synchronize()
    wf = w.copy()
    wf.data = from_bf16(to_bf16(w.data)).astype(np.float64)
    xf = from_bf16(to_bf16(x)).astype(np.float64)
    want, scale = 2.0 * (wf @ xf.T).T, 2.0 * (abs(wf) @ xf.T).T
    # (float32 sums of exact products, in any order, twice)
    assert np.all(np.abs(nat.read("y") - want) <= (n_pre + 64) * 2.0**-23 * scale + 1e-30)
    nat.close()


@pytest.mark.parametrize("graph_steps", [0, 4])
def test_kernels_side_by_side(graph_steps):
    nat = L.NativeNet(0)
    nat.initialize(1.0)
    for name in "abc":
        nat.create(name, np.zeros(1000, np.int32))
    head = "".join(f"__constant__ int* anb_p_{n};\n" for n in "abc")
    body = 'extern "C" __global__ void k{0}() {{ const int i = blockIdx.x * blockDim.x + threadIdx.x; if (i < 1000) {1}; }}\n'
    nat.load_module(head + body.format("a", "anb_p_a[i] += i") + body.format("b", "anb_p_b[i] += 2 * i")
                    + body.format("c", "anb_p_c[i] += anb_p_a[i] + anb_p_b[i]"), [])
    nat.plan([("ka", 4, 256, 0, 1), ("kb", 4, 256, 0, 1), ("kc", 4, 256, 0)])
    nat.set_pdl(False)                        # (kernels without griddepcontrol.wait)
    nat.set_graph_steps(graph_steps)
    nat.run(9)
    nat.synchronize()
    i = np.arange(1000)
    assert np.array_equal(nat.read("a"), 9 * i) and np.array_equal(nat.read("b"), 18 * i)
    assert np.array_equal(nat.read("c"), 3 * i * sum(range(1, 10)))
    nat.close()
