"""Which matrices the automatic storage format lays out in panels instead of
CSR: the edges of the rule."""
import numpy as np
import pytest
import scipy.sparse as sp

from annarchy_b200.generator import formats as F


def _m(n_post, n_pre, lens):
    lens = np.asarray(lens, dtype=np.int64)
    indptr = np.concatenate([[0], np.cumsum(lens)])
    return sp.csr_matrix((np.ones(indptr[-1], np.float32), np.zeros(indptr[-1], np.int32), indptr),
                         shape=(n_post, n_pre))


@pytest.mark.parametrize("n_post,n_pre,lens,want", [
    (1024, 16384, [1024] * 1024, True),                        # 2**20 synapses
    (1024, 16384, [1024] * 1023 + [1023], False),              # one less
    (2**18, 16384 * 2, [4] * 2**18, True),
    (2**18, 16384 * 3, [4] * 2**18, False),                    # 1.33 per row and panel
    (4096, 16384, [300] * 4095 + [16384], False),              # a row with a CTA of its own
    (8192, 16384, [4096] * 8192, True),                        # 2**25
    (8193, 16384, [4096] * 8193, False)])
def test_edges(n_post, n_pre, lens, want):
    assert bool(F.panels_pay(_m(n_post, n_pre, lens))) == want
