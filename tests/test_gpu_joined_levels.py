"""Several tree levels in one launch: root fronts of the largest register
variant (97 to 144 rows), which a first factorization, with a launch per
level, gives to the shared-memory algorithm; and values under which a front
outgrows what the launch was sized for by the factorization before, so that
the factorization stops inside the launch and runs again."""

import numpy as np
import pytest

from amigo_b200.sparse_ldl import CSRMat, OrderingType, SparseLDL
from amigo_b200.workloads import csr_from_coo

pytestmark = pytest.mark.gpu

# growth of the pivoting (ustab = 0.01) below 1e4 at these sizes
BERR = 1e-10


def _sym(rng, n):
    m = rng.standard_normal((n, n))
    return m + m.T


def _solver(a, pattern):
    n = a.shape[0]
    r, c = np.nonzero(pattern)
    rowp, cols, _ = csr_from_coo(n, r, c, np.ones(len(r)))
    rows = np.repeat(np.arange(n), np.diff(rowp))
    mat = CSRMat(n, n, rowp, cols, a[rows, cols])
    return SparseLDL(mat, order=OrderingType.NATURAL), mat, rows, cols


def _factor_solve(ldl, a, b):
    before = ldl.launch_count()
    assert ldl.factor() == 0
    launches = ldl.launch_count() - before
    ev = np.linalg.eigvalsh(a)
    assert tuple(ldl.get_inertia()) == (int((ev > 0).sum()), int((ev < 0).sum()))
    x = np.asfortranarray(b.copy())
    ldl.solve(x)
    scale = np.abs(a).sum(axis=1).max() * np.abs(x).max() + np.abs(b).max()
    assert np.abs(a @ x - b).max() <= BERR * scale
    return x, launches


@pytest.mark.parametrize("sep", [97, 128, 143, 144])
def test_root_of_the_largest_variant(sep):
    """Small fronts under a Bunch-Kaufman root with zeros on its diagonal."""
    rng = np.random.default_rng(sep)
    nb, blk, touch = 4, 3, 5
    n = nb * blk + sep
    a = np.zeros((n, n))
    a[nb * blk:, nb * blk:] = _sym(rng, sep)
    z = np.arange(nb * blk, n, 3)
    a[z, z] = 0.0
    for q in range(nb):
        d = np.arange(q * blk, (q + 1) * blk)
        t = nb * blk + rng.choice(sep, touch, replace=False)
        a[np.ix_(d, d)] = _sym(rng, blk) + 30.0 * np.eye(blk)
        c = rng.standard_normal((touch, blk))
        a[np.ix_(t, d)] = c
        a[np.ix_(d, t)] = c.T
    pattern = a != 0.0
    pattern[nb * blk:, nb * blk:] = True
    ldl, *_ = _solver(a, pattern)
    b = rng.standard_normal((n, 2))
    first, _ = _factor_solve(ldl, a, b)
    assert ldl.stats()["max_front"] == sep
    again, launches = _factor_solve(ldl, a, b)
    assert launches == 1
    assert np.array_equal(first, again)


def _arrow(rng, nb, blk, sep, top, delays):
    """Blocks, their separator, and a few variables on top of it. With
    `delays` no block candidate passes the threshold test in its own front."""
    n = nb * blk + sep + top
    a = np.zeros((n, n))
    s, t = slice(nb * blk, nb * blk + sep), slice(nb * blk + sep, n)
    for q in range(nb):
        d = slice(q * blk, (q + 1) * blk)
        a[d, d] = 1e-9 * _sym(rng, blk) if delays else _sym(rng, blk) + 50.0 * np.eye(blk)
        c = rng.standard_normal((sep, blk))
        a[s, d] = c
        a[d, s] = c.T
    a[s, s] = _sym(rng, sep) + 50.0 * np.eye(sep)
    c = rng.standard_normal((top, sep))
    a[t, s] = c
    a[s, t] = c.T
    a[t, t] = _sym(rng, top) + 50.0 * np.eye(top)
    return a


@pytest.mark.parametrize("nb,blk,sep,top", [(3, 10, 40, 4), (4, 9, 70, 3),  # within 144 rows
                                            (2, 36, 80, 6), (3, 30, 100, 2)])  # beyond
def test_a_front_outgrows_the_launch(nb, blk, sep, top):
    rng = np.random.default_rng(blk + sep)
    plain = _arrow(rng, nb, blk, sep, top, False)
    delaying = _arrow(rng, nb, blk, sep, top, True)
    pattern = plain != 0.0
    b = rng.standard_normal((plain.shape[0], 2))
    ldl, mat, rows, cols = _solver(plain, pattern)
    first, _ = _factor_solve(ldl, plain, b)
    again, launches = _factor_solve(ldl, plain, b)
    small = ldl.stats()["max_front"]
    assert launches == 1 and np.array_equal(first, again)
    mat.vals = delaying[rows, cols]
    grown, repeated = _factor_solve(ldl, delaying, b)
    assert ldl.stats()["max_front"] == nb * blk + sep + top > small + max(8, small // 4)
    assert repeated > launches
    fresh, *_ = _solver(delaying, pattern)
    assert np.array_equal(grown, _factor_solve(fresh, delaying, b)[0])
    mat.vals = plain[rows, cols]
    assert np.array_equal(_factor_solve(ldl, plain, b)[0], first)
