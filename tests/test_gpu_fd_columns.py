"""Forward-difference columns by perturbed field (stress, velocity, pressure,
restore residue) against the oracle, bit for bit: element counts around the
kinds' runs (9, 14, 28) and their common 252, every model and form, with and
without Re and stress diffusion, elements with a restore residue among
others, with and without the arclength column."""
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


def _check(nx, ny, phys, residue=0, rtol=0.0):
    mesh = M.rect_mesh(nx, ny, distort=0.1)
    TL, EU = S.seeded_state(mesh.xyz, phys, 7 * nx + ny)
    rng = np.random.default_rng(1)
    for f, n in zip(rng.integers(0, 6, residue), rng.integers(0, mesh.nnodes, residue)):
        TL[f, n] = np.nextafter(1.0, 0.0)            # x + eps lies in the next binade: (x + eps) - eps != x
    rp, ci = P.build_pattern(mesh.element_nodes(), mesh.nnodes, phys.nex)
    asm = V.BulkAssembler(mesh, phys, rp, ci)
    b, v = asm.set_equations_bulk(TL, EU, "NRP")
    bo, vo = O.assemble(phys, mesh.conn, mesh.xyz, TL, EU if phys.nex else np.zeros(0), rp, ci)
    if rtol:
        assert np.max(np.abs(b - bo)) <= 1e-12 * np.max(np.abs(bo))
        assert np.max(np.abs(v - vo)) <= rtol * np.max(np.abs(vo))
    else:
        assert np.array_equal(b, bo) and np.array_equal(v, vo)
    # the Jacobian alone (no residual requested): the same values
    v2 = np.zeros_like(v)
    asm.assemble(TL, EU if phys.nex else np.zeros(1), V.VEFEM_JAC_FD64, None, v2)
    assert np.array_equal(v2, v)
    asm.close()


@pytest.mark.parametrize("nx,ny", [(1, 1), (4, 2), (3, 3), (5, 2), (13, 1), (7, 2), (5, 3), (9, 3), (7, 4), (29, 1),
                                   (14, 18), (23, 11), (32, 19), (29, 21)])
@pytest.mark.parametrize("form,nex", [("SQRT", 1), ("T", 0)])
def test_partial_runs(nx, ny, form, nex):
    _check(nx, ny, S.giesekus(0.1, 0.5, 0.59, form, nex=nex))


# models with exp(): host and device exp() may differ in the last bit, as on the large meshes
@pytest.mark.parametrize("model,ve,rtol", [("L-PTT", 0.02, 0.0), ("m-L-PTT", 0.05, 0.0), ("e-PTT", 0.05, 1e-6),
                                           ("m-e-PTT", 0.05, 1e-6), ("FENE-CR", 40.0, 0.0), ("FENE-P", 40.0, 0.0),
                                           ("GIESEKUS", 0.2, 0.0)])
@pytest.mark.parametrize("form", ["T", "SQRT"])
@pytest.mark.parametrize("re,df", [(0.0, 0.0), (0.7, 0.0), (0.0, 0.01), (0.7, 0.01)])
def test_models(model, ve, rtol, form, re, df):
    phys = S.Physics(model=model, form=form, WiN=0.4, Wi0=0.4, BvN=0.59, VeN=ve, ReN=re, DfN=df, nex=1)
    _check(6, 5, phys, rtol=rtol)


@pytest.mark.parametrize("form", ["T", "SQRT"])
@pytest.mark.parametrize("residue", [1, 5, 60])
def test_restore_residue_beside_clean_elements(form, residue):
    _check(13, 7, S.oldroyd_b(0.5, 0.59, form, nex=1), residue=residue)


@pytest.mark.parametrize("residue", [3, 700])
def test_restore_residue_on_a_mesh_of_several_waves(residue):
    _check(31, 20, S.oldroyd_b(0.5, 0.59, "SQRT", nex=1), residue=residue)
