"""The predictor's network at sizes that end inside its 16 x 8 tiles and k-steps:
gradients against the oracle (1e-4 of each array's largest entry, as for the
predictor's own sizes), and training in one call, which replays eight
iterations at a time, against the same iterations one call each, bit for bit."""
import numpy as np
import pytest

from oracle.mlp_ref import MLPRef
from ve_flow_around_cylinder_fortran_gb300 import build as B
from ve_flow_around_cylinder_fortran_gb300 import vefem as V

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    B.build()
    V.load()


@pytest.mark.parametrize("inp,out,width,hidden,n", [(1, 1, 1, 1, 1), (17, 5, 33, 1, 16), (98, 32, 256, 3, 17),
                                                    (7, 9, 64, 2, 131), (15, 8, 72, 4, 40)])
def test_sizes(inp, out, width, hidden, n):
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, inp)).astype(np.float32)
    T = rng.standard_normal((n, out)).astype(np.float32)
    nets = [V.MLP(inp, out, width=width, hidden=hidden, seed=4) for _ in range(2)]
    ref = MLPRef(inp, out, width=width, hidden=hidden)
    ref.init_params(4)
    loss, g = nets[0].loss_grad(X, T)
    lr_, gr = ref.loss_grad(X, T)
    assert abs(loss - lr_) <= 1e-5 * lr_
    o = 0
    for i, m in ref.layers:
        for size in (i * m, m):
            assert np.max(np.abs(g[o:o + size] - gr[o:o + size])) <= 1e-4 * np.max(np.abs(gr[o:o + size]))
            o += size
    for iters in (1, 7, 8, 19):
        a = nets[0].train(X, T, iters, 1e-3)
        for _ in range(iters):
            b = nets[1].train(X, T, 1, 1e-3)
        assert a == b and np.array_equal(nets[0].get_params(), nets[1].get_params())
    for net in nets:
        net.close()
