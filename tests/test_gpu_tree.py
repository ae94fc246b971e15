"""The tree elimination (csrc/vefem_tree.cu) on Jacobians the library
assembles: small meshes whose fronts end inside and at the 16-pivot steps and
64-wide tiles, with and without the border, with delayed pressures, against
SuperLU and against the panel elimination."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

from ve_flow_around_cylinder_fortran_gb300 import build as B
from ve_flow_around_cylinder_fortran_gb300 import frontal as FR
from ve_flow_around_cylinder_fortran_gb300 import linsolve as LS
from ve_flow_around_cylinder_fortran_gb300 import mesh as M
from ve_flow_around_cylinder_fortran_gb300 import newton as N
from ve_flow_around_cylinder_fortran_gb300 import pattern as P
from ve_flow_around_cylinder_fortran_gb300 import state as S
from ve_flow_around_cylinder_fortran_gb300 import vefem as V

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    B.build()
    V.load()


def _system(nel, nex, seed):
    mesh = M.build_cylinder_mesh(nel, exact=False)
    phys = S.oldroyd_b(0.3, 0.59, "SQRT", nex=nex)
    rp, ci = P.build_pattern(mesh.element_nodes(), mesh.nnodes, nex)
    asm = V.BulkAssembler(mesh, phys, rp, ci, outlet_edges=True)
    rows, values = N.boundary_conditions(mesh, phys)
    TL, EU = N.initial_state(mesh, phys)
    TL = TL + 0.01 * (S.seeded_state(mesh.xyz, phys, seed)[0] - TL)
    b, vals = N.DeviceAssembly(asm, rows, values, "exact64", True)(TL, EU, True)
    asm.close()
    if nex:
        t = np.random.default_rng(seed).standard_normal(len(rp) - 1)
        vals[rp[-2]:] = t / np.linalg.norm(t)
    return mesh, rp, ci, vals, b, sp.csr_matrix((vals, ci, rp), shape=(len(rp) - 1,) * 2)


@pytest.mark.parametrize("nel,nex,delay", [(40, 1, False), (61, 0, False), (300, 1, True), (523, 0, True),
                                           (523, 1, False), (1150, 1, False)])
def test_tree_matches_superlu_and_panels(nel, nex, delay):
    mesh, rp, ci, vals, b, A = _system(nel, nex, nel)
    lu = FR.FrontalLU(rp, ci, mesh, delay_pressure=delay).factor(vals)
    assert lu.tree and lu.mode == "native" and 0.0 < lu.min_pivot <= 1.0
    x = lu.solve(b)
    ref = LS.SparseLU(rp, ci, mesh).factor(vals).solve(b)
    assert lu.refinements == 0 and lu.solve_path == 2
    assert np.linalg.norm(A @ x - b) <= 1e-10 * np.linalg.norm(b)
    assert np.linalg.norm(x - ref) <= 1e-9 * np.linalg.norm(ref)
    panels = FR.FrontalLU(rp, ci, mesh, panel=6).factor(vals)
    assert not panels.tree and np.linalg.norm(panels.solve(b) - ref) <= 1e-9 * np.linalg.norm(ref)
    # another matrix in between, then the first again: the same bits
    other = vals.copy()
    other[:rp[-2 if nex else -1]] *= 1.5
    lu.factor(torch.from_numpy(other).cuda())
    assert np.linalg.norm(lu.solve(b) - x) > 0.1 * np.linalg.norm(x)
    assert np.array_equal(lu.factor(vals).solve(b), x)
    lu.close()
    panels.close()


def test_singular_front_is_refused():
    mesh, rp, ci, vals, b, A = _system(61, 1, 0)
    k = int(mesh.boundary_nodes["Wall"][3]) * 6
    vals[rp[k]:rp[k + 1]] = 0.0
    vals[rp[k + 1] - 1] = 1.0                            # only the border column
    lu = FR.FrontalLU(rp, ci, mesh).factor(vals)
    A = sp.csr_matrix((vals, ci, rp), shape=A.shape)
    x = lu.solve(b)
    assert lu.resymbolised and lu.pivoted_factorisations == 2 and lu.fallbacks == 1
    assert np.linalg.norm(A @ x - b) <= 1e-10 * np.linalg.norm(b)
    lu.close()
