"""A variable that is coupled to no other and has no number on the diagonal is
a zero pivot of its root front; the solution at the other variables stays what
it is without it."""

import numpy as np
import pytest

from amigo_b200.sparse_ldl import CSRMat, OrderingType, SparseLDL
from amigo_b200.workloads import dense_to_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [6, 40, 90, 140])
def test_isolated_nan_in_a_root_front(n):
    at = 0  # eliminated first: no earlier pivot's back substitution meets it
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    a = a + a.T
    a[at, :] = a[:, at] = 0.0
    a[at, at] = 1.0
    rowp, cols, _ = dense_to_csr(np.ones((n, n)))
    rows = np.repeat(np.arange(n), n)
    b = rng.standard_normal(n)
    xs = []
    for d in (1.0, np.nan):
        a[at, at] = d
        ldl = SparseLDL(CSRMat(n, n, rowp, cols, a[rows, cols]), order=OrderingType.NATURAL)
        x = b.copy()
        for _ in range(2):  # before and after the sizes are known
            assert ldl.factor() == 0
            x = b.copy()
            ldl.solve(x)
        xs.append(x)
    keep = np.arange(n) != at
    assert np.isnan(xs[1][at])
    # the zero pivot comes in the same place of the order, and updates nothing
    assert np.array_equal(xs[0][keep], xs[1][keep])
