"""The tree's way to the pivoted panels: a matrix whose pivots the tree refuses,
before and after the pressures are delayed, and that pivoting inside a panel
factorises; a second one through the same panels; and back to the tree."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

from ve_flow_around_cylinder_fortran_gb300 import frontal as FR
from ve_flow_around_cylinder_fortran_gb300 import linsolve as LS
from test_gpu_tree import _built, _system  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nel,nex", [(61, 1), (300, 0)])
def test_refused_twice_then_pivoted_then_native(nel, nex):
    mesh, rp, ci, vals, b, A = _system(nel, nex, nel)
    lu = FR.FrontalLU(rp, ci, mesh, pivot_tol=0.9)       # no relative pivot is above this everywhere
    other = vals.copy()
    other[:rp[-2 if nex else -1]] *= 1.5
    for v, refused in ((vals, 2), (other, 3)):           # the pressures are delayed once
        lu.factor(torch.from_numpy(v).cuda())
        assert lu.mode == "pivoted" and lu.fallbacks == 0 and lu.resymbolised
        assert lu.pivoted_factorisations == refused
        A = sp.csr_matrix((v, ci, rp), shape=A.shape)
        ref = LS.SparseLU(rp, ci, mesh).factor(v).solve(b)
        for x in (lu.solve(b), lu.solve(torch.from_numpy(b).cuda()).cpu().numpy(),
                  lu.precondition(torch.from_numpy(b).cuda()).cpu().numpy()):
            assert np.linalg.norm(A @ x - b) <= 1e-10 * np.linalg.norm(b)
            assert np.linalg.norm(x - ref) <= 1e-9 * np.linalg.norm(ref)
    lu.pivot_tol = 1e-12
    x = lu.factor(vals).solve(b)
    A = sp.csr_matrix((vals, ci, rp), shape=A.shape)
    assert lu.mode == "native" and lu.pivoted_factorisations == 3 and lu.fallbacks == 0
    assert np.linalg.norm(A @ x - b) <= 1e-10 * np.linalg.norm(b)
    lu.close()
