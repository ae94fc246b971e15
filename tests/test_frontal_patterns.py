"""Patterns with entries between nodes that share no element.  The panels' fronts
hold many of them, the fronts of a nested dissection (made of elements' nodes)
fewer: such a pattern goes to the panels, as it did before the dissection was
the default."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla

from ve_flow_around_cylinder_fortran_gb300 import frontal as FR
from ve_flow_around_cylinder_fortran_gb300 import mesh as M
from ve_flow_around_cylinder_fortran_gb300 import pattern as P

torch = pytest.importorskip("torch")


def _wide_pattern(nel, nex, macro):
    """AIJ pattern of a mesh with couplings, besides the elements' own, among nine
    nodes of every ``macro`` elements in order of x."""
    mesh = M.build_cylinder_mesh(nel, exact=False)
    en = mesh.element_nodes()
    order = np.argsort(mesh.xyz[0][en].mean(axis=1), kind="stable")
    runs = [np.unique(en[order[k:k + macro]]) for k in range(0, len(order), macro)]
    far = np.array([r[np.linspace(0, len(r) - 1, 9).astype(int)] for r in runs])
    return mesh, *P.build_pattern(np.concatenate([en, far]), mesh.nnodes, nex)


@pytest.mark.parametrize("nel,nex,macro,tree", [(60, 1, 4, False), (150, 0, 4, False), (60, 1, 1, True), (150, 0, 1, True)])
def test_entries_outside_the_dissection(monkeypatch, nel, nex, macro, tree):
    mesh, rp, ci = _wide_pattern(nel, nex, macro)
    made = []
    monkeypatch.setattr(FR.FrontalLU, "_create_tree", lambda self: made.append("tree"))
    monkeypatch.setattr(FR.FrontalLU, "_create_native", lambda self: made.append("panels"))
    lu = FR.FrontalLU(rp, ci, mesh, device="cpu")
    lu.tree, lu.method, lu.G = True, "native", 4             # the state of a solver on a CUDA device
    lu._analyse(mesh.element_nodes())
    assert made == (["tree"] if tree else ["panels"]) and lu.tree == tree
    if tree:
        return
    assert lu.G == FR.default_panel(mesh.nel)
    N = len(rp) - 1
    rows = np.repeat(np.arange(N), np.diff(rp))
    rng = np.random.default_rng(nel)
    v = np.where(rows == ci, 40.0, 0.0) + 0.1 * rng.standard_normal(len(ci))
    b = rng.standard_normal(N)
    lu.method = "pivoted"                                    # the same panels, without the library
    x = lu.factor(v).solve(b)
    ref = spla.spsolve(sp.csr_matrix((v, ci, rp), shape=(N, N)).tocsc(), b)
    assert np.linalg.norm(x - ref) <= 1e-9 * np.linalg.norm(ref) and lu.fallbacks == 0
