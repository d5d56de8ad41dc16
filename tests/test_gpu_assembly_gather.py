"""The assembly gather: entries with no, one, two and many contributions at
sizes around a CTA's share (512 entries), bit for bit the sequential sums, and
the factorization from element blocks through the same plan."""

import numpy as np
import pytest

from amigo_b200.assembly import CSRAssembly
from amigo_b200.sparse_ldl import CSRMat, OrderingType, SparseLDL, Vector
from amigo_b200.workloads import csr_from_coo

pytestmark = pytest.mark.gpu


def _pattern(n, conn, extra, rng):
    r = np.concatenate([np.repeat(c, c.shape[1], axis=1).ravel() for c in conn] +
                       [rng.integers(0, n, extra)])
    c = np.concatenate([np.tile(c, (1, c.shape[1])).ravel() for c in conn] +
                       [rng.integers(0, n, extra)])
    rowp, cols, _ = csr_from_coo(n, np.concatenate([r, c]), np.concatenate([c, r]),
                                 np.ones(2 * len(r)))
    return rowp, cols


@pytest.mark.parametrize("n,shapes", [(1, ((1, 1),)), (22, ((3, 2),)), (23, ((40, 3), (5, 1))),
                                      (160, ((300, 4), (90, 2))), (700, ((900, 5), (60, 9)))])
def test_gather_is_the_sequential_sum(n, shapes):
    import torch

    rng = np.random.default_rng(n)
    conn = [np.stack([rng.choice(n, m, replace=False) for _ in range(ne)]) for ne, m in shapes]
    rowp, cols = _pattern(n, conn, n // 2, rng)  # some entries without a contribution
    blocks = []
    for ne, m in shapes:
        b = rng.standard_normal((ne, m, m))
        blocks.append(b + b.transpose(0, 2, 1) + 4.0 * m * np.eye(m))
    want = np.zeros(len(cols))
    for c, b in zip(conn, blocks):
        for e in range(c.shape[0]):
            for j in range(c.shape[1]):
                row = slice(rowp[c[e, j]], rowp[c[e, j] + 1])
                at = rowp[c[e, j]] + np.searchsorted(cols[row], c[e])
                want[at] += b[e, j]
    asm = CSRAssembly(rowp, cols, conn)
    dev = torch.device("cuda")
    flat = torch.as_tensor(np.concatenate([b.ravel() for b in blocks]), device=dev)
    vals = asm.values(flat)
    assert np.array_equal(vals.cpu().numpy(), want)
    diag = torch.full((n,), 3.0, dtype=torch.float64, device=dev)
    xs = []
    for elements in (False, True):
        ldl = SparseLDL(CSRMat(n, n, rowp, cols, vals), order=OrderingType.AMD)
        if elements:
            assert ldl.factor_elements(asm, flat, Vector(diag)) == 0
        else:
            assert ldl.factor(Vector(diag)) == 0
        x = torch.ones(n, dtype=torch.float64, device=dev)
        ldl.solve(x)
        xs.append(x.cpu().numpy())
    assert np.array_equal(xs[0], xs[1])
