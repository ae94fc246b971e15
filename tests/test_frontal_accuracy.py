"""Accuracy that ``FrontalLU.solve`` owes to the tolerance it is given.  The sweep
of the tree elimination leaves so small a residual that a check alone asks for
no refinement; a caller with a tolerance near rounding level gets one all the
same where the panel elimination's sweeps needed it to pass, on all but the
smallest meshes."""
import numpy as np
import pytest

from ve_flow_around_cylinder_fortran_gb300 import frontal as FR
from test_linsolve import _jacobian

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("nel,tol,refine,steps", [(270, 1e-14, 3, 1), (270, 1e-12, 1, 1), (270, 9e-11, 3, 1),
                                                  (270, 1e-14, 0, 0), (270, 1e-10, 3, 0), (270, 1e-8, 3, 0),
                                                  (60, 1.9e-15, 3, 1), (60, 1e-14, 3, 0), (60, 1e-10, 3, 0)])
@pytest.mark.parametrize("tree", [True, False])
def test_refinement_by_tolerance(monkeypatch, tree, nel, tol, refine, steps):
    mesh, rp, ci, v, b = _jacobian(nel, 1)
    N = len(rp) - 1
    rows = np.repeat(np.arange(N), np.diff(rp))
    v = np.where(rows == ci, 8.0, 0.0) + 0.01 * np.random.default_rng(1).standard_normal(len(v))
    lu = FR.FrontalLU(rp, ci, mesh, device="cpu", check_tol=tol, refine=refine).factor(v)
    if tree:                                              # the state of a solver on a CUDA device
        lu.tree, lu.mode = True, "native"
    sweep, rng, delta = lu._sweep_pivoted, np.random.default_rng(2), 2.0 ** -50

    def inexact(r):                                       # relative error delta in every component
        return sweep(r) * torch.from_numpy(1.0 + delta * rng.choice([-1.0, 1.0], N))

    monkeypatch.setattr(lu, "_sweep", inexact)
    for k in range(3):
        x_true = rng.standard_normal(N)
        rhs = np.zeros(N, np.longdouble)
        np.add.at(rhs, rows, v.astype(np.longdouble) * x_true[ci])
        x = lu.solve(rhs.astype(float))
        err = np.linalg.norm(x - x_true) / np.linalg.norm(x_true)
        assert lu.refinements == (steps * (k + 1) if tree else 0) and lu.fallbacks == 0
        # diagonal 8, rows of at most 300 others of 0.01: what rounding leaves is below 2^-52
        assert err <= 2.0 ** -52 if lu.refinements else 2.0 ** -51 <= err <= 2.0 ** -49
