"""One assembly plan shared by threads that each drive a handle of their own
on a stream of their own: the plan's upload happens once, whoever comes first,
and everybody's values and factors are those of a single thread."""

import threading

import numpy as np
import pytest
import torch

from amigo_b200.assembly import CSRAssembly
from amigo_b200.sparse_ldl import CSRMat, OrderingType, SparseLDL, Vector
from tests.test_gpu_assembly_gather import _pattern

pytestmark = pytest.mark.gpu

THREADS = 4


def _one(asm, rowp, cols, flat, diag, start, out, q):
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        start.wait()
        vals = asm.values(flat)
        ldl = SparseLDL(CSRMat(len(diag), len(diag), rowp, cols, vals), order=OrderingType.AMD)
        for _ in range(3):
            ldl.factor_elements(asm, flat, Vector(diag))
            x = torch.ones_like(diag)
            ldl.solve(x)
        stream.synchronize()
        out[q] = (vals.cpu().numpy(), x.cpu().numpy())


@pytest.mark.parametrize("n,shapes", [(23, ((40, 3), (5, 1))), (900, ((1500, 5), (60, 9)))])
def test_shared_plan(n, shapes):
    rng = np.random.default_rng(n)
    conn = [np.stack([rng.choice(n, m, replace=False) for _ in range(ne)]) for ne, m in shapes]
    rowp, cols = _pattern(n, conn, n // 2, rng)
    blocks = []
    for ne, m in shapes:
        b = rng.standard_normal((ne, m, m))
        blocks.append(b + b.transpose(0, 2, 1) + 4.0 * m * np.eye(m))
    flat = torch.as_tensor(np.concatenate([b.ravel() for b in blocks]), device="cuda")
    diag = torch.full((n,), 3.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ready = threading.Barrier(1)
    want = {}
    _one(CSRAssembly(rowp, cols, conn), rowp, cols, flat, diag, ready, want, 0)
    for _ in range(5):
        asm = CSRAssembly(rowp, cols, conn)  # not on the device yet
        start = threading.Barrier(THREADS)
        out = {}
        ts = [threading.Thread(target=_one, args=(asm, rowp, cols, flat, diag, start, out, q))
              for q in range(THREADS)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        assert sorted(out) == list(range(THREADS))
        for got in out.values():
            assert np.array_equal(got[0], want[0][0]) and np.array_equal(got[1], want[0][1])


def test_elements_before_the_plan_is_on_the_device():
    rng = np.random.default_rng(0)
    conn = [np.stack([rng.choice(20, 3, replace=False) for _ in range(30)])]
    rowp, cols = _pattern(20, conn, 4, rng)
    asm = CSRAssembly(rowp, cols, conn)
    flat = torch.zeros(asm.nvals, dtype=torch.float64, device="cuda")
    ldl = SparseLDL(CSRMat(20, 20, rowp, cols, np.ones(len(cols))), order=OrderingType.AMD)
    st = ldl._lib.b200ldl_factor_elements(ldl._h, asm._h, flat.data_ptr(), None)
    assert st == -1 and b"no assembly plan" in ldl._lib.b200ldl_last_error(ldl._h)
