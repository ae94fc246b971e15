"""Calls whose input buffers are overwritten from one call to the next, many
times over: every result has the bits of the first call on the same values.  A
kernel that begins while its predecessors run may not read what they, or those
before them, left in a cache."""
import numpy as np
import pytest
import torch

from ve_flow_around_cylinder_fortran_gb300 import build as B
from ve_flow_around_cylinder_fortran_gb300 import frontal as FR
from ve_flow_around_cylinder_fortran_gb300 import mesh as M
from ve_flow_around_cylinder_fortran_gb300 import pattern as P
from ve_flow_around_cylinder_fortran_gb300 import state as S
from ve_flow_around_cylinder_fortran_gb300 import vefem as V

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    B.build()
    V.load()


@pytest.mark.parametrize("nel", [300, 520, 700, 2000])
def test_forward_difference(nel):
    mesh = M.build_cylinder_mesh(nel, exact=False)
    phys = S.oldroyd_b(0.5, 0.59, "SQRT", nex=1)
    rp, ci = P.build_pattern(mesh.element_nodes(), mesh.nnodes, 1)
    asm = V.BulkAssembler(mesh, phys, rp, ci)
    states = [torch.from_numpy(S.seeded_state(mesh.xyz, phys, s)[0]).cuda() for s in (1, 2, 3)]
    TL, EU = torch.empty_like(states[0]), torch.ones(1, dtype=torch.float64, device="cuda")
    first = {}
    for call in range(24):
        k = call * 7 % 3
        TL.copy_(states[k])
        EU.fill_(1.0 + 0.25 * k)
        b = torch.zeros(asm.N, dtype=torch.float64, device="cuda")
        v = torch.zeros(asm.nnz, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        asm.assemble(TL, EU, V.VEFEM_RESIDUAL | V.VEFEM_JAC_FD64 | V.VEFEM_ZERO_FIRST, b, v, on_device=True)
        torch.cuda.synchronize()
        fb, fv = first.setdefault(k, (b, v))
        assert torch.equal(b, fb) and torch.equal(v, fv)
    asm.close()


@pytest.mark.parametrize("nel", [300, 1150])
def test_factorisation(nel):
    from test_gpu_tree import _system
    mesh, rp, ci, vals, b, _ = _system(nel, 1, nel)
    lu = FR.FrontalLU(rp, ci, mesh)
    matrices = [torch.from_numpy(vals).cuda()]
    for scale in (1.5, -0.75):
        matrices.append(matrices[0].clone())
        matrices[-1][:int(rp[-2])] *= scale
    rhs = torch.from_numpy(b).cuda()
    v, first = torch.empty_like(matrices[0]), {}
    for call in range(45):
        k = call * 7 % 3
        v.copy_(matrices[k])
        lu.factor(v)
        x = lu._sweep(rhs)
        factors, fx = first.setdefault(k, (lu.buf.clone(), x))
        assert lu.mode == "native" and torch.equal(lu.buf, factors) and torch.equal(x, fx)
    lu.close()


@pytest.mark.parametrize("rows", [3, 40, 300])
def test_training(rows):
    """The predictor's network: iterations of one call, whose kernels begin while
    others run, and one call per iteration."""
    rng = np.random.default_rng(rows)
    X = rng.standard_normal((rows, 98)).astype(np.float32)
    T = rng.standard_normal((rows, 32)).astype(np.float32)
    one, many = (V.MLP(98, 32, width=256, hidden=3, seed=1) for _ in range(2))
    for iters in (64, 21):
        a = one.train(X, T, iters, 1e-3)
        for _ in range(iters):
            b = many.train(X, T, 1, 1e-3)
        assert a == b and np.array_equal(one.get_params(), many.get_params())
    one.close()
    many.close()
