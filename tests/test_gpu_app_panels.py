"""The blocked panels with a-posteriori tests (fronts above 144 rows re-planned
from a pivot record): fronts at the edges of a panel (32), a tile (64) and the
row chunks (256), delays that move candidates within and beyond the block,
fronts that run out of candidates, several fronts per level, 2x2 pivots."""

import numpy as np
import pytest

from amigo_b200.sparse_ldl import CSRMat, OrderingType, SparseLDL, Vector
from amigo_b200.workloads import csr_from_coo, hex_elasticity_kkt, plane_stress_kkt

pytestmark = pytest.mark.gpu


def _check(rowp, cols, vals0, vals, diag, inertia, matvec, norm, order, seed):
    """Record at vals0, then factor vals; threshold pivoting (ustab = 0.01)
    grows entries by well below 1e3, hence the backward error."""
    n = len(rowp) - 1
    mat = CSRMat(n, n, rowp, cols, vals0)
    ldl = SparseLDL(mat, order=order)
    d = None if diag is None else Vector(diag)
    assert ldl.factor(d) == 0
    ldl.reuse_pivot_order()
    mat.vals = vals
    b = np.random.default_rng(seed).standard_normal(n)
    xs = []
    for _ in range(2):
        assert ldl.factor(d) == 0
        assert tuple(ldl.get_inertia()) == inertia
        x = b.copy()
        ldl.solve(x)
        xs.append(x)
    assert np.abs(matvec(xs[0]) - b).max() <= 1e-11 * (norm * np.abs(xs[0]).max() + 1.0)
    assert np.array_equal(xs[0], xs[1])
    return ldl


@pytest.mark.parametrize("blk,sep", [(40, 105), (100, 60), (150, 44), (97, 160), (128, 129),
                                     (200, 200), (31, 400), (290, 31)])
def test_blocks_with_a_separator(blk, sep):
    """Saddle-point blocks sharing a separator, recorded at other values: the
    small leading entries change, so that recorded pivots fail and are
    delayed."""
    rng = np.random.default_rng(blk + 7 * sep)
    nb = 3
    n = nb * blk + sep
    a = np.zeros((n, n))
    s = slice(nb * blk, n)
    for q in range(nb):
        d = slice(q * blk, (q + 1) * blk)
        m = rng.standard_normal((blk, blk))
        m = m + m.T
        m[: blk // 3, : blk // 3] *= 1e-6
        a[d, d] = m
        c = rng.standard_normal((sep, blk))
        a[s, d] = c
        a[d, s] = c.T
    m = rng.standard_normal((sep, sep))
    a[s, s] = m + m.T
    p = rng.standard_normal((n, n))
    a1 = a * (1.0 + 0.3 * (p + p.T))
    r, c = np.nonzero(a)
    rowp, cols, _ = csr_from_coo(n, r, c, a[r, c])
    rr = np.repeat(np.arange(n), np.diff(rowp))
    ev = np.linalg.eigvalsh(a1)
    _check(rowp, cols, a[rr, cols], a1[rr, cols], None,
           (int((ev > 0).sum()), int((ev < 0).sum())), lambda x: a1 @ x,
           np.abs(a1).sum(axis=1).max(), OrderingType.NATURAL, blk)


@pytest.mark.parametrize("make", [lambda: plane_stress_kkt(31, seed=5), lambda: plane_stress_kkt(47, seed=6),
                                  lambda: hex_elasticity_kkt(5, seed=7),
                                  lambda: hex_elasticity_kkt(7, seed=8)],
                         ids=["plane_31", "plane_47", "hex_5", "hex_7"])
def test_meshes_with_a_neighbouring_record(make):
    s = make()
    rng = np.random.default_rng(1)
    r = np.repeat(np.arange(s.n, dtype=np.int64), np.diff(s.rowp))
    pos = np.searchsorted(r * s.n + s.cols, s.cols.astype(np.int64) * s.n + r)
    f = rng.standard_normal(s.nnz)
    near = s.vals * (1.0 + 0.02 * (f + f[pos]))
    ldl = _check(s.rowp, s.cols, near, s.vals, s.diag, s.expected_inertia, s.matvec, s.inf_norm(),
                 OrderingType.AMD, 2)
    assert ldl.work()["app_panels"] > 0
