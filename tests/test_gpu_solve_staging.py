"""Supernodes whose factor columns just fit the shared memory of the solves
(40 KB: 5,120 doubles), and just not: roots, fronts with contribution rows, and
a launch in which a large front leaves no room for it."""

import numpy as np
import pytest

from amigo_b200.sparse_ldl import CSRMat, OrderingType, SparseLDL
from amigo_b200.workloads import csr_from_coo

pytestmark = pytest.mark.gpu


def _arrow(blk, sep):
    """Two dense blocks and a dense separator (fronts of blk + sep rows)."""
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


# (f | 1) * pivots: 71 x 71 fits, 73 x 72 does not; 81 x 63 fits, 81 x 64 does not
@pytest.mark.parametrize("blk,sep", [(0, 71), (0, 72), (63, 17), (64, 16), (30, 60), (40, 860),
                                     (40, 960)])
def test_at_the_edge_of_the_room(blk, sep):
    a = _arrow(blk, sep)
    n = a.shape[0]
    r, c = np.nonzero(a)
    rowp, cols, vals = csr_from_coo(n, r, c, a[r, c])
    ldl = SparseLDL(CSRMat(n, n, rowp, cols, vals), order=OrderingType.NATURAL)
    assert ldl.factor() == 0
    b = np.random.default_rng(1).standard_normal((n, 9))
    one = np.empty((n, 9), order="F")
    for q in range(9):
        x = b[:, q].copy()
        ldl.solve(x)
        one[:, q] = x
    # growth of threshold pivoting (ustab = 0.01) below 1e4 at these sizes
    scale = np.abs(a).sum(axis=1).max() * np.abs(one).max() + np.abs(b).max()
    assert np.abs(a @ one - b).max() <= 1e-10 * scale
    for k in (2, 3, 8, 9):
        x = np.asfortranarray(b[:, :k].copy())
        ldl.solve(x)
        assert np.array_equal(x, one[:, :k])
