"""The residual kernels by mesh size (an element over a CTA, three over a CTA,
seven per CTA, batched work items) against the oracle, bit for bit, where one
kernel hands over to the next and where the last CTA is not full."""
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


def _case(nx, ny, form, re, df):
    mesh = M.rect_mesh(nx, ny, distort=0.1)
    phys = S.Physics(model="GIESEKUS", form=form, WiN=0.5, Wi0=0.5, BvN=0.59, VeN=0.1, ReN=re, DfN=df, nex=1)
    TL, EU = S.seeded_state(mesh.xyz, phys, nx * ny)
    return mesh, phys, TL, EU, P.build_pattern(mesh.element_nodes(), mesh.nnodes, 1)


@pytest.mark.parametrize("nx,ny", [(1, 1), (32, 19), (29, 21), (38, 24), (83, 11), (153, 6)])
@pytest.mark.parametrize("form,re,df", [("SQRT", 0.0, 0.0), ("T", 0.0, 0.0), ("SQRT", 1.0, 0.01), ("T", 1.0, 0.0)])
def test_residual_by_size(nx, ny, form, re, df):
    mesh, phys, TL, EU, (rp, ci) = _case(nx, ny, form, re, df)
    asm = V.BulkAssembler(mesh, phys, rp, ci)
    b, _ = asm.set_equations_bulk(TL, EU, "MNR")
    ref, _ = O.assemble(phys, mesh.conn, mesh.xyz, TL, EU, rp, ci)
    assert np.array_equal(b, ref)
    asm.close()
    bt = V.BatchAssembler([mesh, mesh], [phys, phys], [(rp, ci)] * 2)
    bs = [np.zeros(len(rp) - 1) for _ in range(2)]
    bt.assemble([TL, TL], [EU, EU], V.VEFEM_RESIDUAL | V.VEFEM_ZERO_FIRST, bs, None)
    assert np.array_equal(bs[0], ref) and np.array_equal(bs[1], ref)
    bt.close()
