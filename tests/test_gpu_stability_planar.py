"""The two routes of the stability assembly against the oracle, 1e-12 of the
largest entry: planar base states (pairs of in-plane and out-of-plane unknowns
only) for every constitutive model, with and without Re and stress diffusion,
element counts that end inside a block, a pattern with entries outside the
element blocks; and a base state out of the plane (the general kernel)."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import oracle as O
from ve_flow_around_cylinder_fortran_gb300 import build as B_
from ve_flow_around_cylinder_fortran_gb300 import mesh as M
from ve_flow_around_cylinder_fortran_gb300 import pattern as P
from ve_flow_around_cylinder_fortran_gb300 import state as S
from ve_flow_around_cylinder_fortran_gb300 import vefem as V

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    B_.build()
    V.load()


def _check(mesh, phys, TLb, asm, kws, kz=True):
    rp, ci = asm.stability_pattern()
    flags = V.VEFEM_ZERO_FIRST | (0 if kz else V.VEFEM_STAB_AS_WRITTEN)
    fill = [np.full(len(ci), 7.0) for _ in kws]              # ZERO_FIRST overwrites it
    As, B = asm.stability_assemble(TLb, kws, flags, As=fill, B=np.full(len(ci), 7.0))
    en = mesh.element_nodes()
    N = mesh.nnodes * 10
    inod, ieq, jnod, jeq = np.meshgrid(np.arange(9), np.arange(10), np.arange(9), np.arange(10), indexing="ij")
    rows, cols = (en[:, jnod] * 10 + jeq).reshape(-1), (en[:, inod] * 10 + ieq).reshape(-1)
    for k, a in zip(kws, As):
        _, _, Ao, Bo = O.stability_elements(phys, mesh.conn, mesh.xyz, TLb, np.zeros_like(TLb), k, kz=kz)
        for got, ref in ((a, Ao), (B, Bo)):
            R = sp.csr_matrix((ref.reshape(-1), (rows, cols)), shape=(N, N))
            assert abs(sp.csr_matrix((got, ci, rp), shape=(N, N)) - R).max() <= 1e-12 * abs(R).max()
    return As, B


def _base(mesh, phys, planar=True, seed=2):
    TL, _ = S.seeded_state(mesh.xyz, phys, seed=seed)
    TLb = np.zeros((10, mesh.nnodes))
    TLb[0:2], TLb[3:7] = TL[0:2], TL[2:6]
    if not planar:
        rng = np.random.default_rng(5)
        for f in (2, 7, 8, 9):
            TLb[f] = 0.05 * rng.standard_normal(mesh.nnodes)
    return TLb


@pytest.mark.parametrize("model,ve", [("L-PTT", 0.0), ("m-L-PTT", 0.05), ("e-PTT", 0.05), ("m-e-PTT", 0.05),
                                      ("FENE-CR", 40.0), ("FENE-P", 40.0), ("GIESEKUS", 0.2)])
@pytest.mark.parametrize("re,df,planar", [(0.0, 0.0, True), (0.7, 0.01, True), (0.7, 0.0, False)])
def test_models(model, ve, re, df, planar):
    mesh = M.build_cylinder_mesh(43, exact=False)
    phys = S.Physics(model=model, form="T", WiN=0.5, Wi0=0.5, BvN=0.59, VeN=ve, ReN=re, DfN=df, nex=0)
    rp, ci = P.build_pattern(mesh.element_nodes(), mesh.nnodes, 0)
    asm = V.BulkAssembler(mesh, phys, rp, ci)
    _check(mesh, phys, _base(mesh, phys, planar), asm, [0.0, 1.3, -2.0])
    asm.close()


@pytest.mark.parametrize("nx,ny", [(1, 1), (2, 7), (3, 5)])
def test_sizes_both_routes_on_one_context(nx, ny):
    mesh = M.rect_mesh(nx, ny)
    phys = S.oldroyd_b(0.7, 0.59, "T", nex=0)
    rp, ci = P.build_pattern(mesh.element_nodes(), mesh.nnodes, 0)
    asm = V.BulkAssembler(mesh, phys, rp, ci)
    a = _check(mesh, phys, _base(mesh, phys), asm, [0.9])
    _check(mesh, phys, _base(mesh, phys, planar=False), asm, [0.9, 2.0])
    b = _check(mesh, phys, _base(mesh, phys), asm, [0.9])
    assert np.array_equal(a[0][0], b[0][0]) and np.array_equal(a[1], b[1])
    _check(mesh, phys, _base(mesh, phys), asm, [2.0], kz=False)
    asm.close()


def test_pattern_with_entries_outside_the_blocks():
    mesh = M.rect_mesh(4, 3)
    phys = S.oldroyd_b(0.7, 0.59, "T", nex=0)
    en = mesh.element_nodes()
    far = np.linspace(0, mesh.nnodes - 1, 9).astype(en.dtype)   # couples nodes that share no element
    rp, ci = P.build_pattern(np.concatenate([en, far[None]]), mesh.nnodes, 0)
    asm = V.BulkAssembler(mesh, phys, rp, ci)
    assert len(asm.stability_pattern()[1]) > 100 * len(np.unique(
        np.repeat(en, 9, axis=1).ravel() * mesh.nnodes + np.tile(en, (1, 9)).ravel()))
    _check(mesh, phys, _base(mesh, phys), asm, [0.0, 1.1])
    asm.close()
