"""The block ILU(0) factorization (sixteen lanes a row) against NumPy: the
first BiCGSTAB iterate of the adjoint solve is two preconditioner
applications, so it depends on every block of both factors.  The row order is
the solver's: reverse Cuthill-McKee of the renumbered cells."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from conftest import assemble_jt, desc_of, developed_state, small_mesh
from oracle import cpu

pytestmark = pytest.mark.gpu


def _rcm(nbr):
    """BFS from a pseudo-peripheral cell, neighbours by (degree, number),
    reversed; nbr[c]: the cells next to c."""
    def bfs(root):
        out, lvl = [root], {root: 0}
        for u in out:
            for v in sorted((v for v in set(nbr[u]) if v not in lvl), key=lambda v: (len(nbr[v]), v)):
                lvl[v] = lvl[u] + 1
                out.append(v)
        return out, lvl
    order, placed = [], set()
    for start in range(len(nbr)):
        if start in placed:
            continue
        root, depth = start, -1
        for _ in range(4):
            comp, lvl = bfs(root)
            d = lvl[comp[-1]]
            if d <= depth:
                break
            depth, root = d, comp[-1]
            for r in reversed(comp):
                if lvl[r] == d and len(nbr[r]) < len(nbr[root]):
                    root = r
        comp, _ = bfs(root)
        placed.update(comp)
        order += comp
    return order[::-1]


def _ilu0(A, order):
    """Rows {cell: 4x4 block} -> (rows with L and U, inverse diagonals)."""
    pos = {c: i for i, c in enumerate(order)}
    F, Dinv = [{j: b.copy() for j, b in row.items()} for row in A], {}
    for i in order:
        for k in sorted((k for k in F[i] if pos[k] < pos[i]), key=pos.get):
            F[i][k] = F[i][k] @ Dinv[k]
            for j in F[k]:
                if pos[j] > pos[k] and j in F[i]:
                    F[i][j] = F[i][j] - F[i][k] @ F[k][j]
        Dinv[i] = np.linalg.inv(F[i][i])
    return F, Dinv, pos


def _first_iterate(J, b, nbr, order):
    nc = len(nbr)
    D = J.toarray().reshape(nc, 4, nc, 4)
    F, Dinv, pos = _ilu0([{j: D[c, :, j, :] for j in [c, *set(nbr[c])]} for c in range(nc)], order)

    def solve(r):
        y = r.reshape(nc, 4).copy()
        for i in order:
            for k in F[i]:
                if pos[k] < pos[i]:
                    y[i] -= F[i][k] @ y[k]
        for i in reversed(order):
            for j in F[i]:
                if pos[j] > pos[i]:
                    y[i] -= F[i][j] @ y[j]
            y[i] = Dinv[i] @ y[i]
        return y.ravel()

    ph = solve(b)
    v = J @ ph
    alpha = (b @ b) / (b @ v)
    sv = b - alpha * v
    sh = solve(sv)
    t = J @ sh
    return alpha * ph + (t @ sv) / (t @ t) * sh


@pytest.mark.parametrize("n_surface,n_layers,triangles", [(9, 3, True), (13, 5, False), (24, 8, True), (33, 9, False)])
def test_first_iterate_is_that_of_the_numpy_factors(n_surface, n_layers, triangles):
    from optimisation2forme_b200 import HostMesh, SimulationParams, Solver
    from optimisation2forme_b200 import _lib
    p = SimulationParams(viscosity=1.8e-5, inflow_velocity=0.6, aoa_deg=2.0, cfl_number=0.5, final_time=10.0,
                         limiter_k=5.0, verbosity=0)
    m = small_mesh(triangles=triangles, n_surface=n_surface, n_layers=n_layers, seed=4)
    hm = HostMesh(desc=desc_of(m))
    o = cpu.Oracle(hm, p)
    with Solver(p, desc=desc_of(m)) as s:
        U = developed_state(s, 50)
        s.compute_residual()
        lam = s.solve_adjoint_system(beta=0.1, tol=1e-30, max_iter=1, raise_on_failure=False)["lambda"]
        new_of_old = np.zeros(s.n_cells, dtype=np.int64)
        assert _lib.lib().o2f_cell_permutation(s._h, new_of_old.ctypes.data_as(C.POINTER(C.c_int64))) == 0
    LR = o.residual(U)["edge_LR"]
    J, b = assemble_jt(o, hm, LR), o.rhs(LR, 0.1)
    nbr = [[] for _ in range(len(new_of_old))]
    for a, c in hm.array("edge_c").reshape(-1, 2):
        if c >= 0:
            nbr[new_of_old[a]].append(int(new_of_old[c]))
            nbr[new_of_old[c]].append(int(new_of_old[a]))
    old_of_new = np.argsort(new_of_old)
    order = [int(old_of_new[c]) for c in _rcm(nbr)]
    nbr = [[int(old_of_new[v]) for v in nbr[new_of_old[c]]] for c in range(len(nbr))]
    want = _first_iterate(J, b, nbr, order)
    # what a rounding of every input (2^-53) does to it, times 1000 for the
    # roundings of the factorization and the products themselves
    rng = np.random.default_rng(1)
    near = J.copy()
    near.data = near.data * (1 + 1.1e-16 * rng.choice([-1, 1], near.data.size))
    moved = _first_iterate(near, b * (1 + 1.1e-16 * rng.choice([-1, 1], b.size)), nbr, order)
    tol = 1000 * np.linalg.norm(moved - want) + 1e-12 * np.linalg.norm(want)
    err = np.linalg.norm(lam - want)
    print(f"\nfirst iterate: relative difference {err / np.linalg.norm(want):.1e}, bound {tol / np.linalg.norm(want):.1e}")
    assert tol <= 1e-3 * np.linalg.norm(want) and err <= tol
