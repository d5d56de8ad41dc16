"""Fronts factored on chip by one CTA: sizes at the edges of the row chunks
(32, 64, 96) and of the on-chip limit (144), with pivots that stand, that are
interchanged, 2x2 pivots and delays, against numpy. The second factorization
of a pattern runs several tree levels in one launch and has to give the bits
of the first, which runs a level per launch."""

import numpy as np
import pytest

from amigo_b200.sparse_ldl import CSRMat, OrderingType, SparseLDL, Vector
from amigo_b200.workloads import csr_from_coo, dense_to_csr, optimal_control_kkt

pytestmark = pytest.mark.gpu

# |r| <= c n growth eps (|A| |x| + |b|): Bunch-Kaufman and threshold pivoting
# with ustab = 0.01 on these sizes grow entries by well below 1e3
BERR = 1e-11


def _check(rowp, cols, a, nrhs, seed):
    n = a.shape[0]
    vals = a[np.repeat(np.arange(n), np.diff(rowp)), cols]
    ldl = SparseLDL(CSRMat(n, n, rowp, cols, vals), order=OrderingType.NATURAL)
    b = np.random.default_rng(seed).standard_normal((n, nrhs))
    xs = []
    for _ in range(3):
        assert ldl.factor() == 0
        x = np.asfortranarray(b.copy())
        ldl.solve(x)
        xs.append(x)
    ev = np.linalg.eigvalsh(a)
    assert tuple(ldl.get_inertia()) == (int((ev > 0).sum()), int((ev < 0).sum()))
    r = np.abs(a @ xs[0] - b).max()
    assert r <= BERR * (np.abs(a).sum(axis=1).max() * np.abs(xs[0]).max() + np.abs(b).max())
    assert np.array_equal(xs[0], xs[1]) and np.array_equal(xs[0], xs[2])


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 31, 32, 33, 63, 64, 65, 95, 96, 97, 128, 143, 144])
def test_dense_root_front(n):
    """One root front (Bunch-Kaufman); a third of the diagonal is zero, so that
    1x1 pivots at imax and 2x2 pivots occur."""
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    a = a + a.T
    a[np.arange(0, n, 3), np.arange(0, n, 3)] = 0.0 if n > 1 else 1.0
    rowp, cols, _ = dense_to_csr(np.ones((n, n)))
    _check(rowp, cols, a, 2, n)


@pytest.mark.parametrize("sep", [1, 5, 24, 40])
@pytest.mark.parametrize("blk", [3, 8, 27, 56, 88, 103])
def test_blocks_with_a_separator(blk, sep):
    """Dense blocks that share a separator: fronts of blk + sep rows with
    contribution rows; saddle-point blocks with a zero part make candidates
    fail the threshold test (interchanges, 2x2 pivots, delays)."""
    rng = np.random.default_rng(1000 * blk + sep)
    nb = 3
    n = nb * blk + sep
    a = np.zeros((n, n))
    s = slice(nb * blk, n)
    for q in range(nb):
        d = slice(q * blk, (q + 1) * blk)
        m = rng.standard_normal((blk, blk))
        m = m + m.T
        z = blk // 2
        m[:z, :z] *= 1e-9 * (q + 1)
        a[d, d] = m
        c = rng.standard_normal((sep, blk))
        a[s, d] = c
        a[d, s] = c.T
    m = rng.standard_normal((sep, sep))
    a[s, s] = m + m.T + 0.1 * np.eye(sep)
    r, c = np.nonzero(a)
    rowp, cols, _ = csr_from_coo(n, r, c, a[r, c])
    _check(rowp, cols, a, 1, blk)


@pytest.mark.parametrize("N,nx,nu", [(3, 2, 1), (40, 4, 2), (25, 6, 3), (60, 3, 1)])
def test_chain_of_fronts_in_one_launch(N, nx, nu):
    """An optimal-control system's narrow tree: the first factorization, the
    ones after it (one launch for the levels), and a run on another handle's
    values give the same solution bit for bit."""
    s = optimal_control_kkt(N=N, nx=nx, nu=nu, nrhs=3, seed=N)
    ldl = SparseLDL(CSRMat(s.n, s.n, s.rowp, s.cols, s.vals), order=OrderingType.AMD)
    xs = []
    for _ in range(3):
        assert ldl.factor(Vector(s.diag)) == 0
        assert tuple(ldl.get_inertia()) == s.expected_inertia
        x = np.asfortranarray(s.rhs.copy())
        ldl.solve(x)
        xs.append(x)
    r = np.abs(s.matvec(xs[0]) - s.rhs).max()
    assert r <= 1e-12 * (s.inf_norm() * np.abs(xs[0]).max() + np.abs(s.rhs).max())
    assert np.array_equal(xs[0], xs[1]) and np.array_equal(xs[0], xs[2])
