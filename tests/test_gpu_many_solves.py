"""The solves' progress flags start over after 4,096 launches' worth of
right-hand sides: solves before, at and after that give the same bits, also
when that falls inside a call of several launches."""

import numpy as np
import pytest
import torch

from amigo_b200.sparse_ldl import CSRMat, OrderingType, SparseLDL, Vector
from amigo_b200.workloads import optimal_control_kkt, plane_stress_kkt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make", [lambda: optimal_control_kkt(N=12, nrhs=1, seed=2),
                                  lambda: plane_stress_kkt(10, seed=3)], ids=["chain", "plane"])
def test_flags_start_over(make):
    s = make()
    ldl = SparseLDL(CSRMat(s.n, s.n, s.rowp, s.cols, s.vals), order=OrderingType.AMD)
    assert ldl.factor(Vector(s.diag)) == 0
    b = torch.as_tensor(np.random.default_rng(0).standard_normal((17, s.n)), device="cuda")
    want = b.clone()
    ldl.solve(want.t())  # three launches of up to eight columns
    for _ in range(1400):  # 4,200 launches in all
        x = b.clone()
        ldl.solve(x.t())
        assert torch.equal(x, want)
