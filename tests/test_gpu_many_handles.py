"""More handles alive at once than a page of failure words serves (1,024), made,
used and destroyed by several threads, twice over."""

import threading

import numpy as np
import pytest

from amigo_b200.sparse_ldl import CSRMat, OrderingType, SparseLDL, Vector
from amigo_b200.workloads import optimal_control_kkt

pytestmark = pytest.mark.gpu


def test_handles_come_and_go():
    s = optimal_control_kkt(N=3, nx=2, nu=1, nrhs=1, seed=0)
    mat = CSRMat(s.n, s.n, s.rowp, s.cols, s.vals)
    rhs = np.ascontiguousarray(s.rhs.reshape(s.n, -1)[:, 0])

    def solve():
        ldl = SparseLDL(mat, order=OrderingType.AMD)
        assert ldl.factor(Vector(s.diag)) == 0
        x = rhs.copy()
        ldl.solve(x)
        return ldl, x

    want = solve()[1]
    for _ in range(2):
        bad, done = [], []

        def work():
            mine = [solve() for _ in range(280)]
            bad.extend(q for q, (_, x) in enumerate(mine) if not np.array_equal(x, want))
            done.append(len(mine))

        threads = [threading.Thread(target=work) for _ in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert done == [280] * 4 and not bad
