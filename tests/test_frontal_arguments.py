"""What ``FrontalLU.factor`` is given is checked before any of it reaches the
library: the library reads as many values and places as it is told to."""
import numpy as np
import pytest

from ve_flow_around_cylinder_fortran_gb300 import frontal as FR
from test_linsolve import _jacobian

torch = pytest.importorskip("torch")


class _Library:
    """Stands in for the library; takes note of the factorisations it is asked for."""

    def __init__(self):
        self.factored = []

    def vefem_tree_factor(self, handle, vals, dest, nnz, buf, buf_len, stream, tol, min_pivot):
        self.factored.append(nnz)
        return 0

    def vefem_tree_destroy(self, handle):
        pass


@pytest.mark.parametrize("tree", [True, False])
@pytest.mark.parametrize("shape", [lambda n: n - 1, lambda n: n + 1, lambda n: 1, lambda n: (n, 1), lambda n: (2, n)])
@pytest.mark.parametrize("kind", ["host", "tensor"])
def test_values_of_another_shape_are_refused(monkeypatch, tree, shape, kind):
    mesh, rp, ci, v, b = _jacobian(30, 1)
    lu = FR.FrontalLU(rp, ci, mesh, device="cpu")
    if tree:                                             # the state of a solver on a CUDA device
        lu.tree, lu.method, lu._L, lu._handle = True, "native", _Library(), 1
        monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: type("S", (), {"cuda_stream": 0}))
    bad = np.ones(shape(len(v)))
    with pytest.raises(RuntimeError):
        lu.factor(bad if kind == "host" else torch.from_numpy(bad))
    if tree:
        assert lu._L.factored == []
        lu.factor(v)
        assert lu._L.factored == [len(v)]
