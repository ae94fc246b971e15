"""Exact FP64 Jacobian at the mesh sizes where a work item's elements change (one
up to one per SM, two up to two, then three) and up to which the residual goes
first (three per SM): the same bits as in a batch large enough for whole groups,
and within 1e-12 of the oracle's complex-step Jacobian on the smaller ones, also
as a batch of one."""
import numpy as np
import pytest

from oracle import oracle as O
from ve_flow_around_cylinder_fortran_gb300 import build as B
from ve_flow_around_cylinder_fortran_gb300 import mesh as M
from ve_flow_around_cylinder_fortran_gb300 import pattern as P
from ve_flow_around_cylinder_fortran_gb300 import state as S
from ve_flow_around_cylinder_fortran_gb300 import vefem as V

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    B.build()
    V.load()


@pytest.mark.parametrize("nx,ny", [(1, 1), (20, 2), (151, 1), (152, 1), (153, 1), (101, 3), (152, 2), (61, 5), (307, 1), (152, 3), (457, 1)])
@pytest.mark.parametrize("form", ["T", "SQRT"])
def test_items_of_every_size(nx, ny, form):
    mesh = M.rect_mesh(nx, ny, distort=0.1)
    phys = S.giesekus(0.1, 0.5, 0.59, form, nex=1)
    TL, EU = S.seeded_state(mesh.xyz, phys, nx)
    rp, ci = P.build_pattern(mesh.element_nodes(), mesh.nnodes, 1)
    asm = V.BulkAssembler(mesh, phys, rp, ci)
    b, v = asm.set_equations_bulk(TL, EU, "NRP", jacobian="exact64")
    big = M.rect_mesh(90, 8)
    pat = [(rp, ci), P.build_pattern(big.element_nodes(), big.nnodes, 1)]
    meshes, states = [mesh, big], [(TL, EU), S.seeded_state(big.xyz, phys, 1)]
    for n in (2, 1):
        bt = V.BatchAssembler(meshes[:n], [phys] * n, pat[:n])
        bs = [np.zeros(len(p[0]) - 1) for p in pat[:n]]
        vs = [np.zeros(len(p[1])) for p in pat[:n]]
        bt.assemble([s[0] for s in states[:n]], [s[1] for s in states[:n]],
                    V.VEFEM_RESIDUAL | V.VEFEM_JAC_EXACT64 | V.VEFEM_ZERO_FIRST, bs, vs)
        assert np.array_equal(bs[0], b) and np.array_equal(vs[0], v)
        bt.close()
    if nx * ny <= 305:
        bo, vo = O.exact_assemble(phys, mesh.conn, mesh.xyz, TL, EU, rp, ci)
        assert np.max(np.abs(v - vo)) <= 1e-12 * np.max(np.abs(vo))
    asm.close()
