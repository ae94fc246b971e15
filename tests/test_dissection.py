"""Nested-dissection fronts (dissection.py) on the CPU: every unknown is
eliminated once, every pattern entry lies in the front of the first of its two
unknowns, a front's boundary lies in its parent, and eliminating front by front
solves the bordered system."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla

from ve_flow_around_cylinder_fortran_gb300 import dissection as D
from ve_flow_around_cylinder_fortran_gb300 import mesh as M
from ve_flow_around_cylinder_fortran_gb300 import pattern as P


def _tree(nel, nex, leaf, delay):
    mesh = M.build_cylinder_mesh(nel, exact=False)
    en = mesh.element_nodes()
    rp, ci = P.build_pattern(en, mesh.nnodes, nex)
    return D.Tree(en, mesh.xyz[:2][:, en].mean(axis=2), mesh.nnodes, 6, nex, leaf, delay), rp, ci


@pytest.mark.parametrize("nel,nex,leaf,delay", [(40, 1, 4, None), (61, 0, 4, None), (120, 1, 2, 2),
                                                (120, 1, 200, None), (150, 0, 7, 2)])
def test_fronts_cover_the_pattern_and_solve(nel, nex, leaf, delay):
    t, rp, ci = _tree(nel, nex, leaf, delay)
    N = len(rp) - 1
    fronts = [t.ids[t.idx_off[k]:t.idx_off[k + 1]] for k in range(t.nfront)]
    piv = np.concatenate([f[:p] for f, p in zip(fronts, t.p)])
    assert np.array_equal(np.sort(piv), np.arange(N))
    if nex:
        assert all(f[-1] == N - 1 for f in fronts)
    rows = np.repeat(np.arange(N), np.diff(rp))
    q = t.front_of[np.maximum(t.owner[rows], t.owner[ci])]
    rng = np.random.default_rng(0)
    v = rng.standard_normal(len(ci)) * 0.1
    v[rows == ci] += 10.0
    A = sp.csr_matrix((v, ci, rp), shape=(N, N))
    b = rng.standard_normal(N)
    # dense elimination front by front
    y, x, fac, schur = b.copy(), np.zeros(N), [], {}
    order = np.argsort(q, kind="stable")
    ptr = np.searchsorted(q[order], np.arange(t.nfront + 1))
    pos = np.full(N, -1)
    for k in range(t.nfront):
        f, p, h = fronts[k], t.p[k], t.heap[k]
        pos[:] = -1
        pos[f] = np.arange(len(f))
        e = order[ptr[k]:ptr[k + 1]]
        assert (pos[rows[e]] >= 0).all() and (pos[ci[e]] >= 0).all()
        F = np.zeros((len(f), len(f)))
        F[pos[rows[e]], pos[ci[e]]] = v[e]
        for c in (2 * h, 2 * h + 1):
            if c in schur:
                u, S = schur.pop(c)
                assert (pos[u] >= 0).all()
                F[np.ix_(pos[u], pos[u])] += S
        Ai = np.linalg.inv(F[:p, :p])
        X = Ai @ F[:p, p:]
        schur[h] = (f[p:], F[p:, p:] - F[p:, :p] @ X)
        z = Ai @ y[f[:p]]
        y[f[p:]] -= F[p:, :p] @ z
        fac.append((f, p, z, X))
    for f, p, z, X in reversed(fac):
        x[f[:p]] = z - X @ x[f[p:]]
    ref = spla.spsolve(A.tocsc(), b)
    assert np.linalg.norm(x - ref) <= 1e-10 * np.linalg.norm(ref)
