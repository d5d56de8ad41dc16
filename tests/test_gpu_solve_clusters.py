"""Supernodes that take a cluster in the solves (fronts of at least 1024
rows): roots, and with contribution rows, with sizes at the edges of the 32-row
tiles and of the CTAs' shares. A column's bits do not depend on the others or
on the run."""

import numpy as np
import pytest

from amigo_b200.sparse_ldl import CSRMat, OrderingType, SparseLDL
from amigo_b200.workloads import csr_from_coo

pytestmark = pytest.mark.gpu

CLUSTER = 1024  # rows of the smallest front that takes one


def _dense(n):
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    return a + a.T


def _arrow(blk, sep):
    """Two dense blocks coupled to a dense separator."""
    n = 2 * blk + sep
    rng = np.random.default_rng(n)
    a = np.zeros((n, n))
    s = slice(2 * blk, n)
    for q in range(2):
        d = slice(q * blk, (q + 1) * blk)
        m = rng.standard_normal((blk, blk))
        a[d, d] = m + m.T
        c = rng.standard_normal((sep, blk))
        a[s, d] = c
        a[d, s] = c.T
    m = rng.standard_normal((sep, sep))
    a[s, s] = m + m.T
    return a


@pytest.mark.parametrize("a", [_dense(1024), _dense(1055), _arrow(600, 425), _arrow(33, 1100)],
                         ids=["root1024", "root1055", "arrow600-425", "arrow33-1100"])
def test_columns_and_runs(a):
    n = a.shape[0]
    r, c = np.nonzero(a)
    rowp, cols, vals = csr_from_coo(n, r, c, a[r, c])
    ldl = SparseLDL(CSRMat(n, n, rowp, cols, vals), order=OrderingType.NATURAL)
    b = np.random.default_rng(1).standard_normal((n, 9))
    scale = np.abs(a).sum(axis=1).max()
    for reuse in (False, True):
        if reuse:
            ldl.reuse_pivot_order()
        assert ldl.factor() == 0
        assert ldl.stats()["max_front"] >= CLUSTER
        x = np.asfortranarray(b.copy())
        ldl.solve(x)
        # growth of threshold pivoting (ustab = 0.01) below 1e4 at these sizes
        assert np.abs(a @ x - b).max() <= 1e-10 * (scale * np.abs(x).max() + np.abs(b).max())
        for k in (1, 2, 3, 8, 9):
            y = np.asfortranarray(b[:, :k].copy())
            ldl.solve(y)
            assert np.array_equal(y, x[:, :k])
