"""A wait inside a launch that is given up: with a limit of no polls at all the
fronts of a later level find their children unfinished and give up at once.
The kernels end, the call reports it, and the handle works as before."""

import numpy as np
import pytest

from amigo_b200.sparse_ldl import CSRMat, OrderingType, SparseLDL, SparseLDLBatch, Vector
from amigo_b200.workloads import optimal_control_kkt

pytestmark = pytest.mark.gpu

DEFAULT = 1 << 23


def _chain():
    s = optimal_control_kkt(N=60, nrhs=3, seed=1)
    ldl = SparseLDL(CSRMat(s.n, s.n, s.rowp, s.cols, s.vals), order=OrderingType.AMD)
    return ldl, s.diag, s.rhs


def _batch():
    systems = [optimal_control_kkt(N=20 + q, nrhs=1, seed=q) for q in range(40)]
    ldl = SparseLDLBatch([CSRMat(s.n, s.n, s.rowp, s.cols, s.vals) for s in systems],
                         order=OrderingType.AMD)
    return ldl, np.concatenate([s.diag for s in systems]), np.concatenate(
        [s.rhs.reshape(s.n, -1)[:, :1] for s in systems])


def _solve(ldl, rhs):
    x = np.asfortranarray(rhs.copy())
    ldl.solve(x)
    return x


@pytest.mark.parametrize("make", [_chain, _batch], ids=["chain", "batch"])
def test_given_up_and_usable_after(make):
    ldl, diag, rhs = make()
    assert ldl.factor(Vector(diag)) == 0
    assert ldl.factor(Vector(diag)) == 0  # several levels share a launch
    want = _solve(ldl, rhs)
    for _ in range(3):
        ldl.set_wait_limit(0)
        with pytest.raises(RuntimeError, match="were not solved in time"):
            _solve(ldl, rhs)
        ldl.set_wait_limit(DEFAULT)
        assert np.array_equal(_solve(ldl, rhs), want)
        ldl.set_wait_limit(0)
        with pytest.raises(RuntimeError, match="did not complete in time"):
            ldl.factor(Vector(diag))
        with pytest.raises(RuntimeError, match="before a successful factor"):
            _solve(ldl, rhs)
        ldl.set_wait_limit(DEFAULT)
        assert ldl.factor(Vector(diag)) == 0
        assert np.array_equal(_solve(ldl, rhs), want)


def test_bad_limit():
    ldl, _, _ = _chain()
    with pytest.raises(ValueError, match="negative"):
        ldl.set_wait_limit(-1)
