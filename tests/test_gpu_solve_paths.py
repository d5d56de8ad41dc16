"""The solve kernels over the numbers of right-hand sides at the edges of
their variants and launches (1, 2, 4, 8, and chunks of 8 with a remainder),
on systems whose supernodes keep their factor in shared memory, stream it,
and take clusters. Every right-hand side is computed by the same operations
in the same order whatever its neighbours, so the columns solved one at a
time are the same bits."""

import numpy as np
import pytest

from amigo_b200.sparse_ldl import CSRMat, OrderingType, SparseLDL, Vector
from amigo_b200.workloads import optimal_control_kkt, plane_stress_kkt

pytestmark = pytest.mark.gpu


def _systems():
    yield "chain", optimal_control_kkt(N=70, nx=5, nu=2, nrhs=17, seed=2), False
    yield "plane_first", plane_stress_kkt(20, seed=3, nrhs_random=16), False
    yield "plane_reuse", plane_stress_kkt(40, seed=4, nrhs_random=16), True


@pytest.fixture(scope="module", params=list(_systems()), ids=lambda p: p[0])
def factored(request):
    _, s, reuse = request.param
    ldl = SparseLDL(CSRMat(s.n, s.n, s.rowp, s.cols, s.vals), order=OrderingType.AMD)
    assert ldl.factor(Vector(s.diag)) == 0
    if reuse:
        ldl.reuse_pivot_order()
        assert ldl.factor(Vector(s.diag)) == 0
    single = np.empty((s.n, 17), order="F")
    for j in range(17):
        x = s.rhs[:, j].copy()
        ldl.solve(x)
        single[:, j] = x
    return s, ldl, single


@pytest.mark.parametrize("nrhs", [1, 2, 3, 4, 5, 7, 8, 9, 16, 17])
def test_columns_are_independent(factored, nrhs):
    s, ldl, single = factored
    x = np.asfortranarray(s.rhs[:, :nrhs].copy())
    ldl.solve(x)
    assert np.array_equal(x, single[:, :nrhs])
    # backward error of a stable solve (growth below 1e3 at ustab = 0.01)
    r = np.abs(s.matvec(x) - s.rhs[:, :nrhs]).max(axis=0)
    scale = s.inf_norm() * np.abs(x).max(axis=0) + np.abs(s.rhs[:, :nrhs]).max(axis=0)
    assert np.all(r <= 1e-12 * scale)
