"""The exact-Jacobian kernel where its element groups are not full (1 to 9
elements, FP32 and FP64, single and batched) and with Re and stress diffusion,
against the oracle's complex-step Jacobian: FP64 within 1e-12 of the largest
entry, FP32 within 1e-5, as on the large meshes."""
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


def _check(mesh, phys, nex):
    TL, EU = S.seeded_state(mesh.xyz, phys, 3)
    rp, ci = P.build_pattern(mesh.element_nodes(), mesh.nnodes, nex)
    asm = V.BulkAssembler(mesh, phys, rp, ci)
    bo, vo = O.exact_assemble(phys, mesh.conn, mesh.xyz, TL, EU, rp, ci)
    for jac, tol in (("exact64", 1e-12), ("exact32", 1e-5)):
        b, v = asm.set_equations_bulk(TL, EU, "NRP", jacobian=jac)
        assert np.max(np.abs(v - vo)) <= tol * np.max(np.abs(vo)), jac
        bt = V.BatchAssembler([mesh] * 2, [phys] * 2, [(rp, ci)] * 2)
        bs, vs = [np.zeros(len(rp) - 1) for _ in range(2)], [np.zeros_like(v) for _ in range(2)]
        bt.assemble([TL] * 2, [EU if nex else np.zeros(1)] * 2,
                    V.VEFEM_RESIDUAL | V.JACOBIANS[jac] | V.VEFEM_ZERO_FIRST, bs, vs)
        assert all(np.array_equal(x, b) for x in bs) and all(np.array_equal(x, v) for x in vs)
        bt.close()
    asm.close()


@pytest.mark.parametrize("nx,ny", [(1, 1), (2, 1), (3, 1), (2, 2), (5, 1), (3, 3)])
@pytest.mark.parametrize("form,nex", [("SQRT", 1), ("T", 0)])
def test_partial_groups(nx, ny, form, nex):
    _check(M.rect_mesh(nx, ny, distort=0.1), S.giesekus(0.1, 0.5, 0.59, form, nex=nex), nex)


@pytest.mark.parametrize("model,ve", [("L-PTT", 0.02), ("m-L-PTT", 0.05), ("e-PTT", 0.05), ("m-e-PTT", 0.05),
                                      ("FENE-CR", 40.0), ("FENE-P", 40.0), ("GIESEKUS", 0.2)])
@pytest.mark.parametrize("form", ["T", "SQRT"])
@pytest.mark.parametrize("re,df", [(0.7, 0.0), (0.0, 0.01), (0.7, 0.01)])
def test_inertia_and_diffusion(model, ve, form, re, df):
    phys = S.Physics(model=model, form=form, WiN=0.4, Wi0=0.4, BvN=0.59, VeN=ve, ReN=re, DfN=df, nex=1)
    _check(M.rect_mesh(4, 3, distort=0.2), phys, 1)
