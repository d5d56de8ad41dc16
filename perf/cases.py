"""The work that a user of the KKT solver has it do, as cases to be timed.

An interior-point loop holds one solver handle per sparsity pattern and, on
every iteration, factors new values and solves with the factor. The cases
follow that use through the public entry points (``SparseLDL``,
``SparseLDLBatch``, ``kkt_solve``, ``CSRAssembly``) over the workload
families of ``amigo_b200.workloads``:

- ``oc``: one optimal-control system (small fronts, a long narrow tree);
- ``batch``: many optimal-control systems of uneven size in one handle;
- ``grad``: a batch of equal systems, solved and differentiated;
- ``plane``: the 2D plane-stress system (fronts up to thousands of rows);
- ``hex``: the 3D elasticity system with one dense constraint row;
- ``assembly``: the KKT values gathered from element Hessian blocks.

``order`` is "first" for a handle's first factorization (the reference's
pivot sequence) and "reuse" for a refactorization on the pivot order that a
neighbouring iterate recorded. ``solve`` cases keep the factor and solve.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from amigo_b200.assembly import CSRAssembly
from amigo_b200.autograd import kkt_solve
from amigo_b200.sparse_ldl import CSRMat, OrderingType, SparseLDL, SparseLDLBatch, Vector
from amigo_b200.workloads import (
    hex_elasticity_kkt,
    optimal_control_kkt,
    plane_stress_kkt,
)


def listed():
    return [
        # the smallest call: a short-horizon controller re-solved on line
        {"name": "oc_n50", "kind": "oc", "N": 50, "nx": 4, "nu": 2, "nrhs": 1, "host": False},
        # the plain workload: N = 1000 nodes, eight right-hand sides
        {"name": "oc_n1000", "kind": "oc", "N": 1000, "nx": 4, "nu": 2, "nrhs": 8, "host": False},
        # the same size from host arrays, as a CPU program's solver plugin calls it
        {"name": "oc_n1000_host", "kind": "oc", "N": 1000, "nx": 4, "nu": 2, "nrhs": 1,
         "host": True},
        # 512 independent systems of 50..400 nodes in one handle
        {"name": "batch_512", "kind": "batch", "systems": 512, "nmin": 50, "nmax": 400,
         "nx": 6, "nu": 3},
        # 64 equal systems solved and differentiated (factor, solve, adjoint solve, gradients)
        {"name": "grad_64", "kind": "grad", "systems": 64, "N": 500, "nx": 4, "nu": 2},
        # the first factorization of a mid-size pattern
        {"name": "plane_64_first", "kind": "plane", "nel": 64, "nrhs": 4, "order": "first"},
        # a refactorization of a mid-size pattern
        {"name": "plane_101_reuse", "kind": "plane", "nel": 101, "nrhs": 4, "order": "reuse"},
        # the headline: refactorization and five-column solve of the 256 x 256 mesh
        {"name": "plane_256_reuse", "kind": "plane", "nel": 256, "nrhs": 4, "order": "reuse"},
        # sensitivities on a stored factor: one right-hand side, and eight
        {"name": "plane_128_solve", "kind": "solve", "nel": 128, "nrhs": 0, "refine": False},
        {"name": "plane_128_refine", "kind": "solve", "nel": 128, "nrhs": 7, "refine": True},
        # a 3D pattern with a dense row, refactored
        {"name": "hex_11_reuse", "kind": "hex", "nel": 11, "nrhs": 4, "order": "reuse"},
        # the KKT values of the 256 x 256 mesh from element blocks
        {"name": "assembly_256", "kind": "assembly", "nel": 256},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["oc", "oc", "batch", "grad", "plane", "plane", "plane", "solve", "solve",
                       "hex", "assembly"])
    if kind == "oc":
        return {"kind": "oc", "N": _log(rng, 30, 4000), "nx": rng.randint(2, 6),
                "nu": rng.randint(1, 3), "nrhs": rng.randint(1, 8), "host": rng.random() < 0.3}
    if kind == "batch":
        lo = rng.randint(30, 100)
        return {"kind": "batch", "systems": _log(rng, 8, 512), "nmin": lo,
                "nmax": lo + rng.randint(0, 300), "nx": rng.randint(3, 6),
                "nu": rng.randint(1, 3)}
    if kind == "grad":
        return {"kind": "grad", "systems": _log(rng, 1, 64), "N": _log(rng, 50, 500),
                "nx": rng.randint(3, 6), "nu": rng.randint(1, 3)}
    if kind == "plane":
        order = rng.choice(["first", "reuse", "reuse"])
        return {"kind": "plane", "nel": _log(rng, 16, 100 if order == "first" else 240),
                "nrhs": rng.randint(0, 7), "order": order}
    if kind == "solve":
        return {"kind": "solve", "nel": _log(rng, 24, 180), "nrhs": rng.randint(0, 15),
                "refine": rng.random() < 0.4}
    if kind == "hex":
        return {"kind": "hex", "nel": rng.randint(4, 12), "nrhs": rng.randint(0, 7),
                "order": rng.choice(["first", "reuse", "reuse"])}
    return {"kind": "assembly", "nel": _log(rng, 16, 300)}


# ---------------------------------------------------------------- inputs


def _systems(case, seed):
    """The case's KKT systems (one, or a batch), made from the seed."""
    kind = case["kind"]
    if kind == "oc":
        return [optimal_control_kkt(case["N"], case["nx"], case["nu"], nrhs=case["nrhs"],
                                    seed=seed)]
    if kind == "batch":
        # the sizes belong to the case (batched_optimal_control's for its seed 0)
        sizes = np.random.default_rng(0).integers(case["nmin"], case["nmax"] + 1,
                                                  size=case["systems"])
        rng = np.random.default_rng(seed)
        return [optimal_control_kkt(int(N), case["nx"], case["nu"], nrhs=1, rng=rng)
                for N in sizes]
    if kind == "grad":
        rng = np.random.default_rng(seed)
        return [optimal_control_kkt(case["N"], case["nx"], case["nu"], nrhs=1, rng=rng)
                for _ in range(case["systems"])]
    if kind == "hex":
        return [hex_elasticity_kkt(case["nel"], seed=seed, nrhs_random=case["nrhs"])]
    return [plane_stress_kkt(case["nel"], seed=seed, nrhs_random=case["nrhs"])]


def _neighbour(s, seed):
    """Values of a neighbouring interior-point iterate: the entries scaled
    symmetrically by 1 + 0.01 N(0, 1), Sigma by exp(0.3 N(0, 1))."""
    rng = np.random.default_rng(seed + 1)
    r = np.repeat(np.arange(s.n, dtype=np.int64), np.diff(s.rowp))
    pos = np.searchsorted(r * s.n + s.cols, s.cols.astype(np.int64) * s.n + r)
    f = rng.standard_normal(s.nnz)
    d = s.diag.copy()
    m = d > 0
    d[m] *= np.exp(0.3 * rng.standard_normal(int(m.sum())))
    return s.vals * (1.0 + 0.005 * (f + f[pos])), d


def _mesh(nel):
    """Element variables (8 displacements, density, 8 multipliers) of the
    nel x nel plane-stress mesh and whether they are clamped."""
    nn1 = nel + 1
    ex, ey = np.meshgrid(np.arange(nel), np.arange(nel), indexing="xy")
    n0 = (ex + ey * nn1).ravel()
    nodes = np.stack([n0, n0 + 1, n0 + 1 + nn1, n0 + nn1], axis=1)
    dofs = np.empty((nel * nel, 8), dtype=np.int64)
    dofs[:, 0::2] = 2 * nodes
    dofs[:, 1::2] = 2 * nodes + 1
    off_rho = 2 * nn1 * nn1
    off_lam = off_rho + nel * nel
    rho = off_rho + np.arange(nel * nel, dtype=np.int64)
    return np.concatenate([dofs, rho[:, None], off_lam + dofs], axis=1)


def _blocks(nel, seed, dev):
    """Symmetric element Hessian blocks, [elements, 17, 17]."""
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    b = torch.randn(nel * nel, 17, 17, dtype=torch.float64, device=dev, generator=g)
    return (b + b.transpose(1, 2)).contiguous()


def _cm(a, dev):
    """[n, k] host array as a column-major device tensor."""
    return torch.as_tensor(np.ascontiguousarray(a.T), device=dev).t()


def prepare(case, seed):
    kind = case["kind"]
    dev = torch.device("cuda")
    if kind == "assembly":
        s = plane_stress_kkt(case["nel"], seed=0, nrhs_random=0)
        asm = CSRAssembly(s.rowp, s.cols, [_mesh(case["nel"])])
        return {"kind": kind, "asm": asm, "blocks": _blocks(case["nel"], seed, dev),
                "out": torch.empty(s.nnz, dtype=torch.float64, device=dev)}
    systems = _systems(case, seed)
    if kind in ("batch", "grad"):
        mats = [CSRMat(s.n, s.n, s.rowp, s.cols, s.vals) for s in systems]
        ldl = SparseLDLBatch(mats, order=OrderingType.AMD)
        vals = torch.as_tensor(np.concatenate([s.vals for s in systems]), device=dev)
        diag = torch.as_tensor(np.concatenate([s.diag for s in systems]), device=dev)
        rhs = torch.as_tensor(np.concatenate([s.rhs[:, 0] for s in systems]), device=dev)
        st = {"kind": kind, "ldl": ldl, "vals": vals, "diag": diag, "rhs": rhs}
        if kind == "grad":
            for t in (vals, diag, rhs):
                t.requires_grad_(True)
            st["primal"] = torch.as_tensor(np.concatenate(
                [np.arange(s.n) < s.n_primal for s in systems]).astype(np.float64), device=dev)
        return st
    s = systems[0]
    if kind == "oc" and case["host"]:
        mat = CSRMat(s.n, s.n, s.rowp, s.cols, s.vals)
        return {"kind": "host", "ldl": SparseLDL(mat, order=OrderingType.AMD),
                "diag": Vector(s.diag), "rhs": s.rhs}
    vals = torch.as_tensor(s.vals, device=dev)
    diag = torch.as_tensor(s.diag, device=dev)
    mat = CSRMat(s.n, s.n, s.rowp, s.cols, vals)
    ldl = SparseLDL(mat, order=OrderingType.AMD)
    if case.get("order") == "reuse" or kind == "solve":
        nv, nd = _neighbour(s, seed)
        mat.vals = torch.as_tensor(nv, device=dev)
        ldl.factor(Vector(torch.as_tensor(nd, device=dev)))
        ldl.reuse_pivot_order()
        mat.vals = vals
    if kind == "solve":
        ldl.factor(Vector(diag))
    return {"kind": kind, "ldl": ldl, "diag": Vector(diag), "rhs": _cm(s.rhs, dev),
            "refine": case.get("refine", False)}


def run(state):
    kind = state["kind"]
    if kind == "assembly":
        return state["asm"].values(state["blocks"], out=state["out"])
    ldl = state["ldl"]
    if kind == "batch":
        ldl.factor(state["diag"], values=state["vals"])
        x = state["rhs"].clone()
        ldl.solve(x)
        return {"x": x, "inertia": np.array(ldl.system_inertia())}
    if kind == "grad":
        vals, diag, rhs = state["vals"], state["diag"], state["rhs"]
        x = kkt_solve(ldl, vals, diag, rhs)
        loss = 0.5 * (state["primal"] * x * x).sum()
        gv, gd, gb = torch.autograd.grad(loss, (vals, diag, rhs))
        return {"x": x.detach(), "gvals": gv, "gdiag": gd, "grhs": gb}
    if kind == "host":
        ldl.factor(state["diag"])
        x = np.array(state["rhs"], order="F")
        ldl.solve(x)
        return {"x": x, "inertia": np.array(ldl.get_inertia())}
    if kind == "solve":
        if state["refine"]:
            x, berr, iters = ldl.solve_refine(state["rhs"], diagonal=state["diag"])
            return {"x": x}
        x = state["rhs"].clone()
        ldl.solve(x)
        return {"x": x}
    ldl.factor(state["diag"])
    x = state["rhs"].clone()
    ldl.solve(x)
    return {"x": x, "inertia": np.array(ldl.get_inertia())}


# ---------------------------------------------------------------- work


def _factor_work(s):
    """(entries of L, factorization flops) of the symbolic structure."""
    ldl = SparseLDL(CSRMat(s.n, s.n, s.rowp, s.cols, s.vals), order=OrderingType.AMD)
    sym = ldl.symbolic()
    p = np.diff(sym["node_ptr"]).astype(np.float64)
    f = p + np.diff(sym["contrib_ptr"])
    ldl.close()
    entries = float(np.sum(p * f - p * (p - 1) / 2))
    # sum of r^2 for r = f - 1 down to f - p
    sq = lambda m: (m - 1) * m * (2 * m - 1) / 6  # noqa: E731
    return entries, float(np.sum(sq(f) - sq(f - p)))


def work(case):
    if case["kind"] == "assembly":
        ne = case["nel"] ** 2
        nnz = 93 * ne
        return {"bytes": 8.0 * 289 * ne + 8.0 * nnz, "flops": 289.0 * ne}
    if case["kind"] == "batch":
        s = optimal_control_kkt((case["nmin"] + case["nmax"]) // 2, case["nx"], case["nu"], 1)
        count = case["systems"]
    elif case["kind"] == "grad":
        s, count = optimal_control_kkt(case["N"], case["nx"], case["nu"], 1), case["systems"]
    else:
        s, count = _systems(case, 0)[0], 1
    nrhs = s.rhs.shape[1]
    entries, flops = _factor_work(s)
    solve = 4.0 * entries * nrhs
    if case["kind"] == "solve":
        more = 12.0 * s.nnz if case["refine"] else 0.0
        return {"bytes": 8.0 * entries + 16.0 * s.n * nrhs + more,
                "flops": solve + (2.0 * s.nnz * nrhs if case["refine"] else 0.0)}
    moved = 8.0 * (s.nnz + s.n + 2 * s.n * nrhs)
    if case["kind"] == "grad":
        moved, solve = moved + 8.0 * (s.nnz + 2 * s.n), 2 * solve + 2.0 * s.nnz
    return {"bytes": count * moved, "flops": count * (flops + solve)}


# ---------------------------------------------------------------- 64-bit values


def _groups(case, s):
    """(group, position in the group) of every variable, so that couplings
    run only inside a group and between neighbouring groups."""
    if case["kind"] in ("oc", "batch", "grad"):
        m = case["nx"] + case["nu"]
        N = s.n_primal // m
        stage = np.concatenate([np.repeat(np.arange(N), m),
                                np.repeat(np.arange(N - 1), case["nx"])])
        g = stage // 8
    elif case["kind"] == "hex":
        g = np.zeros(s.n, dtype=np.int64)
    else:
        nel = case["nel"]
        row = np.repeat(np.arange(nel + 1), 2 * (nel + 1))
        g = np.concatenate([row, np.repeat(np.arange(nel), nel), row])
    order = np.argsort(g, kind="stable")
    start = np.searchsorted(g[order], np.arange(g.max() + 1))
    at = np.empty(s.n, dtype=np.int64)
    at[order] = np.arange(s.n) - start[g[order]]
    return g, at


def _matrix(systems, dev):
    """COO rows, columns and values of the block-diagonal matrix."""
    off = np.concatenate([[0], np.cumsum([s.n for s in systems])])
    rows, cols, vals = [], [], []
    for s, o in zip(systems, off):
        rows += [np.repeat(np.arange(s.n), np.diff(s.rowp)) + o, np.arange(s.n) + o]
        cols += [s.cols + o, np.arange(s.n) + o]
        vals += [s.vals, s.diag]
    put = lambda a, t: torch.as_tensor(np.concatenate(a).astype(t), device=dev)  # noqa: E731
    return put(rows, np.int64), put(cols, np.int64), put(vals, np.float64)


class _Dense64:
    """Block-tridiagonal LU of the systems by dense blocks, with residual
    corrections: an independent 64-bit solver."""

    def __init__(self, case, systems, dev):
        r, c, v = self.rcv = _matrix(systems, dev)
        gp = [_groups(case, s) for s in systems]
        self.n = sum(s.n for s in systems)
        sysid = torch.as_tensor(np.repeat(np.arange(len(systems)), [s.n for s in systems]),
                                device=dev)
        g = torch.as_tensor(np.concatenate([a for a, _ in gp]), device=dev)
        at = torch.as_tensor(np.concatenate([b for _, b in gp]), device=dev)
        S, G, m = len(systems), int(g.max()) + 1, int(at.max()) + 1
        self.shape, self.where = (S, G, m), (sysid * G + g) * m + at
        D = torch.zeros(S * G * m * m, dtype=torch.float64, device=dev)
        E = torch.zeros(S * G * m * m, dtype=torch.float64, device=dev)  # group g+1 rows, g columns
        slot = (self.where[r] * m + at[c])
        same = g[r] == g[c]
        D.index_add_(0, slot[same], v[same])
        low = g[r] == g[c] + 1
        E.index_add_(0, ((sysid[c] * G + g[c])[low] * m + at[r][low]) * m + at[c][low], v[low])
        D, self.E = D.view(S, G, m, m), E.view(S, G, m, m)
        pad = torch.ones(S * G * m, dtype=torch.float64, device=dev)
        pad[self.where] = 0.0
        D.diagonal(dim1=2, dim2=3).add_(pad.view(S, G, m))
        self.lu = []
        for k in range(G):
            a = D[:, k]
            if k:
                low = self.E[:, k - 1]
                a = a - low @ torch.linalg.lu_solve(*self.lu[-1], low.transpose(1, 2))
            self.lu.append(torch.linalg.lu_factor(a))

    def _apply(self, b):
        S, G, m = self.shape
        k = b.shape[1]
        y = torch.zeros(S * G * m, k, dtype=torch.float64, device=b.device)
        y[self.where] = b
        y = y.view(S, G, m, k)
        for q in range(1, G):
            y[:, q] -= self.E[:, q - 1] @ torch.linalg.lu_solve(*self.lu[q - 1], y[:, q - 1])
        for q in range(G - 1, -1, -1):
            t = y[:, q]
            if q + 1 < G:
                t = t - self.E[:, q].transpose(1, 2) @ y[:, q + 1]
            y[:, q] = torch.linalg.lu_solve(*self.lu[q], t)
        return y.view(S * G * m, k)[self.where]

    def solve(self, b):
        r, c, v = self.rcv
        x = self._apply(b)
        for _ in range(3):
            res = b.clone().index_add_(0, r, v[:, None] * x[c], alpha=-1.0)
            x = x + self._apply(res)
        return x


def exact(case, seed):
    kind = case["kind"]
    dev = torch.device("cuda")
    if kind == "assembly":
        s = plane_stress_kkt(case["nel"], seed=0, nrhs_random=0)
        conn = _mesh(case["nel"])
        blocks = _blocks(case["nel"], seed, dev).cpu()
        key = np.repeat(np.arange(s.n, dtype=np.int64), np.diff(s.rowp)) * s.n + s.cols
        want = (conn[:, :, None] * s.n + conn[:, None, :]).ravel()
        pos = np.minimum(np.searchsorted(key, want), s.nnz - 1)
        keep = key[pos] == want
        out = torch.zeros(s.nnz, dtype=torch.float64)
        out.index_add_(0, torch.as_tensor(pos[keep]), blocks.reshape(-1)[torch.as_tensor(keep)])
        return out
    if kind == "hex" and case["nel"] > 11:  # its dense matrix has more than 12,000 rows
        return None
    systems = _systems(case, seed)
    lu = _Dense64(case, systems, dev)
    b = torch.as_tensor(np.concatenate([s.rhs for s in systems]), device=dev)
    x = lu.solve(b)
    if kind == "batch":
        return {"x": x[:, 0], "inertia": None}
    if kind == "grad":
        primal = torch.as_tensor(np.concatenate([np.arange(s.n) < s.n_primal for s in systems]),
                                 device=dev)
        lam = lu.solve(torch.where(primal[:, None], x, torch.zeros_like(x)))
        off = np.concatenate([[0], np.cumsum([s.n for s in systems])])
        r = torch.as_tensor(np.concatenate([np.repeat(np.arange(s.n), np.diff(s.rowp)) + o
                                            for s, o in zip(systems, off)]), device=dev)
        c = torch.as_tensor(np.concatenate([s.cols + o for s, o in zip(systems, off)]),
                            device=dev).long()
        lam, x = lam[:, 0], x[:, 0]
        return {"x": x, "gvals": -lam[r] * x[c], "gdiag": -lam * x, "grhs": lam}
    if kind == "solve":
        return {"x": x}
    if kind == "oc" and case["host"]:
        return {"x": x.cpu().numpy(), "inertia": None}
    return {"x": x, "inertia": None}
